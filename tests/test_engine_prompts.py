"""The engine's tile GEMM with steps of 256 to 1000 rows, one to four 256-wide and 128-wide row and weight tiles: queries, keys and values
into their places, gated products, sums in one and several planes; weight rows and heads that end inside a tile, sizes off the tile's on
every side.  Bars as everywhere for the bf16 format (lm_case.py)."""
import os
import sys

import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import lm_models as M  # noqa: E402
import vupuzen_oracle as V  # noqa: E402
from lm_case import Case  # noqa: E402


@pytest.mark.parametrize("width,mixer,ff", [(1088, ("attention", M.attention(64, 4, 64, 64, 40)), 2056),
                                            (520, ("attention", M.attention(72, 3, 48, 64, 25)), 4100),
                                            (1032, ("retention", M.retention(24, 48, 80, 48, [0.9 + i / 250 for i in range(24)])), 3000)])
def test_prompts(width, mixer, ff, tmp_path):
    cfg = M.config(width, 300, [M.layer(*mixer, ff)], taps=3)
    w = M.weights(cfg, 11)
    c = Case(M.write(tmp_path / "m", cfg, w), V, cfg, w, "bfloat16", max_seqs=2, max_ctx=1008, max_rows=1000)
    toks = c.tokens(1000)
    want = c.oracle(toks)
    for n in (256, 257, 383, 500, 513, 768, 897, 1000):
        c.check(c.run(toks[:n]), want[:n])
    c.model.close()
