"""The convolution of long portions, four rows a block (256 rows and more, up to four taps): portions that end inside a block, inputs
from the step, from the state of the step before and in front of the first token; five taps stay with the other kernel."""
import pytest

import dabevik_oracle as o
from test_gpu_dabevik import TOL, err, load, tokens_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_portions_match_the_oracle(tmp_path, taps, dtype):
    cfg = o.make_config(vocab=70, width=40, taps=taps, max_positions=600, layers=[o.make_layer(4, 2, 16, 16, size=40, keep_first=2, ff=40) for _ in range(2)])
    w = o.make_weights(cfg, 3)
    toks = tokens_for(cfg, 523, 4)
    want = o.forward(cfg, w, toks)
    dec = load(o.save_model(str(tmp_path), cfg, w), dtype, prefill_rows=512)
    for cuts in ([256, 267], [2, 257, 264], [512, 11]):
        dec.reset_sequence(0)
        at = 0
        for c in cuts:
            got = dec.extend(toks[at:at + c], at, list(range(0, c, 3)) + [c - 1])
            assert err(got, want[[at + i for i in list(range(0, c, 3)) + [c - 1]]]) < TOL[dtype], (cuts, at)
            at += c
