"""Scores of mixed heads of portions at head sizes whose queries stay in registers (64 and 128 after padding) and that do not."""
import pytest

import dabevik_oracle as o
import test_gpu_mixed_heads as mixed

pytestmark = pytest.mark.gpu

SIZES = [64, 56, 120, 80, 48]


@pytest.mark.parametrize("dim", SIZES)
def test_scores_of_head_sizes(tmp_path, monkeypatch, dim):
    cfg = o.make_config(vocab=70, width=48, taps=1, layers=mixed.layers((4, 2, dim, 16, 90, 3), (18, 9, dim, 24, 150, 0)))
    monkeypatch.setitem(mixed.MODELS, "size", cfg)
    mixed.test_portions_match_the_oracle(tmp_path, "size", 128)
