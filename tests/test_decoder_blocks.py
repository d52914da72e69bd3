"""Prompts through the operators that write their linear's operand blocks themselves.  Every row of an operator with its linear has the
bits of the operator followed by the linear's own quantization; and one layer of a decoder at the edges of those kernels, its last row
(which sees the others through the first norm's keys and values alone) against the numpy oracle.  Bar on the 2-norm of the last logits: an int8 activation on a boundary may go the other way, which moves the
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


# the same edges row by row: int8 blocks (policy 5 up to 192 rows of a narrow matrix too), fp16 blocks of the tile GEMMs with and without
# rows of padding, K-split counters; one CTA a row and four; K off 32, 8 and 4
@pytest.mark.parametrize("op,k", [(0, 64), (0, 72), (0, 1032), (0, 2048), (1, 40), (1, 3073), (1, 3080), (1, 4864), (1, 6152), (1, 8960),
                                  (1, 9224), (1, 12000)])
@pytest.mark.parametrize("m,n,kernel", [(5, 96, 0), (33, 40, 5), (41, 64, 0), (64, 64, 5), (65, 64, 0), (128, 96, 5), (130, 40, 0), (200, 64, 5),
                                        (257, 320, 5)])
def test_every_row_has_the_bits_of_operator_and_quantization(op, k, m, n, kernel):
    import ctypes as C

    import torch
    import mllm_b200 as mb
    rng = np.random.default_rng(op + k + m)
    wt = mb.W4A32Weights.from_blob(mb.quant_prepack((rng.standard_normal((n, k)) / np.sqrt(k)).astype(np.float32), rng.standard_normal(n).astype(np.float32)))
    dev = lambda a: torch.from_numpy(np.asarray(a, np.float32)).cuda()  # noqa: E731
    a, b, w = dev(rng.standard_normal((m, k)) * 2), dev(rng.standard_normal((m, k))), dev(1 + 0.1 * rng.standard_normal(k))
    a[m // 2], b[m // 2] = 0, 0
    out = []
    for form in (0, 1):
        x, h, y = (torch.full((m, c), float("nan"), device="cuda") for c in (k, k, n))
        ws = torch.full((mb.workspace_size(m, k),), 0x7e, dtype=torch.uint8, device="cuda")
        st = mb.lib().mllmb200_selftest_operator_linear(op, form, a.data_ptr(), b.data_ptr(), w.data_ptr(), 1e-6, m, k, n, wt.tiled.data_ptr(),
                                                        ws.data_ptr(), x.data_ptr(), h.data_ptr(), y.data_ptr(), kernel,
                                                        C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0, mb.status_str(st)
        torch.cuda.synchronize()
        mb.check_device_status()
        out.append((y, h))
    assert torch.isfinite(out[0][0]).all() and torch.equal(out[0][0], out[1][0])
    assert op == 1 or torch.equal(out[0][1], out[1][1])
