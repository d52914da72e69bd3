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


def _attention(q, k, v, sin, cos, form):
    """Output and caches of the prompt attention by itself; q [n, H, D], k and v [n, G, D], sin and cos [n, D / 2]."""
    import ctypes as C
    import mllm_b200 as mb
    import torch
    f = mb.lib().mllmb200_selftest_prompt_attention
    f.argtypes, f.restype = [C.c_void_p] * 3 + [C.c_int] * 4 + [C.c_void_p] * 2 + [C.c_int] + [C.c_void_p] * 4, C.c_int
    n, H, D = q.shape
    G = k.shape[1]
    out, ck, cv = (torch.full(s, float("nan"), device="cuda") for s in ((n, H, D), (G, n, D), (G, n, D)))
    torch.cuda.synchronize()
    st = f(q.data_ptr(), k.data_ptr(), v.data_ptr(), n, H, G, D, sin.data_ptr(), cos.data_ptr(), form, ck.data_ptr(), cv.data_ptr(),
           out.data_ptr(), None)
    assert st == 0, mb.status_str(st)
    mb.check_device_status()
    return out, ck, cv


def _attention64(q, k, v, sin, cos):
    import torch
    q, k, v, sin, cos = (t.double() for t in (q, k, v, sin[:, None], cos[:, None]))
    d = q.shape[2] // 2
    q, k = (torch.cat([x[..., :d] * cos - x[..., d:] * sin, x[..., :d] * sin + x[..., d:] * cos], -1) for x in (q, k))
    later = torch.ones(len(q), len(q), dtype=torch.bool, device="cuda").triu(1)
    out, group = torch.empty_like(q), q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // group].T * q.shape[2] ** -0.5).masked_fill(later, -float("inf"))
        out[:, h] = s.softmax(-1) @ v[:, h // group]
    return out


def _inputs(group, dim, n, seed, kv_heads=2):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn((n, h, dim), device="cuda", generator=g) for h in (group * kv_heads, kv_heads, kv_heads))
    angle = torch.rand((n, dim // 2), device="cuda", generator=g) * 6.2831853
    return q, k, v, angle.sin(), angle.cos()


def _worst_row(out, want):
    return float(((out.double() - want).norm(dim=-1) / want.norm(dim=-1)).max())


# Bar on every row of every head, normal q, k, v: a score is a sum of D products of about 1 / sqrt(D) with D^0.5 of them left
# after cancellation, each off by at most 3 x 2^-22 (two halves, the product of low halves); 3 D / 16 additions truncate by
# 2^-23 of the partial sum each.  That is about 1e-6 of a weight, and the output's sum adds as much: 4e-6.  (Without the low
# halves it is 1e-4 and more; a key too many or too few among 8192 is 1 / 90 of a row's norm.)
BAR = 4e-6


@pytest.mark.gpu
@pytest.mark.parametrize("group,dim", [(1, 64), (6, 128), (7, 64), (8, 128), (5, 128)])
def test_every_row_in_both_forms(group, dim):
    """All rows, so that the causal limit of each is seen: lengths around tiles of 64 positions and of 128 / group tokens, and
    around the length at which the decoder changes form."""
    import torch
    for n in sorted({1, 2, 128 // group, 128 // group + 1, 63, 64, 65, 96, 97, 127, 128, 129, 191, 300}):
        args = _inputs(group, dim, n, 7 * n + group)
        want = _attention64(*args)
        got = {form: _attention(*args, form) for form in (0, 1, 2)}
        for form in (1, 2):
            assert _worst_row(got[form][0], want) <= BAR, (n, form)
        assert torch.equal(got[0][0], got[1 if n <= 96 else 2][0]), n
        for i in (1, 2):
            assert torch.allclose(got[1][i], got[2][i], rtol=2e-7, atol=2e-7)  # (a fused multiply-add here or there)


@pytest.mark.gpu
@pytest.mark.parametrize("group,dim,n", [(6, 128, 4500), (7, 64, 8191)])
def test_every_row_of_a_long_prompt(group, dim, n):
    args = _inputs(group, dim, n, n, kv_heads=1)
    assert _worst_row(_attention(*args, 0)[0], _attention64(*args)) <= BAR


@pytest.mark.gpu
@pytest.mark.parametrize("what,factor", [("k", 3e3), ("v", 3e3), ("k", 5e4), ("v", 5e4), ("v", 1e30), ("v", 1e-30), ("k", float("inf")), ("v", float("inf")),
                                         ("k", float("nan")), ("v", float("nan"))])
@pytest.mark.parametrize("group,dim", [(6, 128), (1, 64)])
def test_a_position_does_not_reach_rows_in_front_of_it(group, dim, what, factor):
    """One position whose key or value has another size than its neighbours, or is no number.  Rows in front of it have the
    accuracy they always have; those that see it are the fp32 form's, bit for bit (a factor of 3000 still fits the tile)."""
    import torch
    n, p = 300, 150
    q, k, v, sin, cos = _inputs(group, dim, n, 11)
    clean = _attention64(q, k, v, sin, cos)
    (k if what == "k" else v)[p, 0] *= factor
    got, fp32 = (_attention(q, k, v, sin, cos, form)[0] for form in (2, 1))
    front = got[:p // 4 * 4]  # (four rows at a time: 0 times infinity)
    assert _worst_row(front, clean[:len(front)]) <= BAR
    if factor != 3e3:  # the heads with that position
        assert torch.equal(got[p:, :group].view(torch.int32), fp32[p:, :group].view(torch.int32))
    assert _worst_row(got[:, group:], clean[:, group:]) <= BAR  # the others
