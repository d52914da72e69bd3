"""The decoder's prompt attention (tensor cores, operands split in two) at the edges of its tiles: 64 cache positions, and
128 / group tokens of a KV head's query heads.  One layer, logits of the last token against the numpy oracle.

Bar: 5e-3 of the logits' rms, the decoder's own.  The embedding is 8 times the size of the attention's output, so that an
activation that falls to the other side of an int8 boundary (at most 1 / 127 of one of >= 64 inputs of a linear) stays
below 1e-3, while a key too many or too few among 300 would show as 8e-3 or more of the rms for most of them."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
from oracle_lib import Oracle  # noqa: E402
from qwen2_oracle import Qwen2Oracle  # noqa: E402
from test_decoder import _gpu_decoder, bind_oracle_linears, make_model  # noqa: E402


def case(group, dim, v_scale):
    cfg = dict(layers=1, hidden=128, q_heads=2 * group, kv_heads=2, head_dim=dim, inter=64, vocab=257, max_ctx=320, eps=1e-6, rope_theta=10000.0)
    w, raw = make_model(cfg, 40 + group)
    w["embedding"] *= 8
    scale = {"v": v_scale, "o": 1 / v_scale}
    raw = [(l, name, (wt * scale.get(name, 1)).astype(np.float32), None if b is None else (b * scale.get(name, 1)).astype(np.float32))
           for l, name, wt, b in raw]
    return cfg, bind_oracle_linears(w, raw, Oracle()), raw


# values beyond fp16's range and below its subnormals as well: every tile brings its own power of two
@pytest.mark.gpu
@pytest.mark.parametrize("group,dim,v_scale", [(1, 64, 1.0), (7, 64, 1e6), (6, 128, 1.0), (8, 128, 1e-9)])
def test_prompt_attention_at_tile_edges(group, dim, v_scale):
    import mllm_b200 as mb
    cfg, w, raw = case(group, dim, v_scale)
    dec, ref = _gpu_decoder(cfg, w, raw), Qwen2Oracle(cfg, w)
    rng, tokens = np.random.default_rng(group), 128 // group
    for n in sorted({1, tokens, tokens + 1, 63, 64, 65, 128, 129, 192, 300}):
        prompt = rng.integers(0, cfg["vocab"], n)
        ref.reset()
        want = ref.forward(list(prompt))
        dec.prefill(prompt)
        got = dec.read(0, 0, want_logits=True)[2]
        mb.check_device_status(dec.stream())
        rms = float(np.sqrt(np.mean(want.astype(np.float64) ** 2)))
        err = float(np.max(np.abs(got - want)))
        assert err <= 5e-3 * rms, (n, err / rms)
    dec.close()
