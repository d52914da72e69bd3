"""Prompts through the operators that write their linear's operand blocks themselves: one layer at the edges of those kernels, against
the numpy oracle.  Bar on the 2-norm of the last logits: an int8 activation on a boundary may go the other way, which moves the
outputs of one linear by up to a quantum of one of its K inputs, 2^-8 of the row's range over sqrt(K); with a handful of those
in a layer 5e-3 (LOGIT_TOL of test_decoder.py, there on the largest difference)."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
from qwen2_oracle import Qwen2Oracle  # noqa: E402
from oracle_lib import Oracle  # noqa: E402
from test_decoder import LOGIT_TOL, _gpu_decoder, bind_oracle_linears, make_model  # noqa: E402


# int8 blocks of one and of uneven blocks of rows, fp16 blocks with and without rows of padding; a thread's 1 to 4 items of the
# feed-forward, widths that are no multiple of 32, of 8 and of 4
@pytest.mark.parametrize("hidden,inter,n", [(64, 40, 5), (72, 3073, 33), (256, 6152, 41), (64, 9224, 9), (64, 12000, 64), (1032, 1184, 70),
                                            (256, 3080, 130), (104, 9218, 200), (2048, 96, 257)])
def test_prompt_blocks(hidden, inter, n):
    cfg = dict(layers=1, hidden=hidden, q_heads=2, kv_heads=1, head_dim=64, inter=inter, vocab=500, max_ctx=n + 8, eps=1e-6, rope_theta=1e4)
    orc = Oracle()
    w, raw = make_model(cfg, hidden + inter)
    bind_oracle_linears(w, raw, orc)
    prompt = np.random.default_rng(n).integers(0, cfg["vocab"], n).tolist()
    want = Qwen2Oracle(cfg, w).generate(prompt, 0)[1][0].astype(np.float64)
    dec = _gpu_decoder(cfg, w, raw)
    dec.prefill(prompt)
    got = dec.read(n - 1, 1, want_logits=True)[2].astype(np.float64)
    assert np.linalg.norm(got - want) <= LOGIT_TOL * np.linalg.norm(want)
