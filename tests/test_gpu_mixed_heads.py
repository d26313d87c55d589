"""Mixed heads of portions at the edges of the kernel that takes all of 17 to 32 heads at once (8 queries a block, pairs of
heads of one key head, 32 keys a tile): fewest and most heads, heads that leave MMA rows empty, one and several key
heads, value sizes that are no whole tiles, windows shorter and longer than a tile, rows that end inside a block."""
import pytest

import dabevik_oracle as o
from test_gpu_dabevik import TOL, err, load, tokens_for

pytestmark = pytest.mark.gpu


def layers(*specs):
    return [o.make_layer(h, kv, d, vd, size=size, keep_first=keep, ff=40) for h, kv, d, vd, size, keep in specs]


MODELS = {
    "eighteen": o.make_config(vocab=90, width=48, taps=1, layers=layers((18, 9, 16, 24, 40, 3), (18, 1, 16, 16, 7, 0))),
    "thirty-two": o.make_config(vocab=90, width=64, taps=2, layers=layers((32, 8, 32, 40, 300, 4), (32, 16, 16, 16, 33, 35))),
    "twenty-six": o.make_config(vocab=70, width=40, taps=1, layers=layers((26, 13, 16, 12, 64, 1))),
    "widest": o.make_config(vocab=70, width=64, taps=1, layers=layers((32, 8, 128, 128, 100, 2))),
    # not these: an odd number of heads per key head, more than 32 heads
    "others": o.make_config(vocab=70, width=48, taps=1, layers=layers((21, 7, 16, 16, 50, 2), (34, 17, 16, 16, 50, 2))),
}


@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("rows", [64, 256])
def test_portions_match_the_oracle(tmp_path, name, rows):
    cfg = MODELS[name]
    w = o.make_weights(cfg, 5)
    toks = tokens_for(cfg, 203, 2)
    want = o.forward(cfg, w, toks)
    dec = load(o.save_model(str(tmp_path), cfg, w), "bfloat16", prefill_rows=rows)
    for cuts in ([203], [16, 17, 100, 70], [41, 162]):
        dec.reset_sequence(0)
        at = 0
        for c in cuts:
            got = dec.extend(toks[at:at + c], at, list(range(c)))
            assert err(got, want[at:at + c]) < TOL["bfloat16"], (cuts, at)
            at += c
