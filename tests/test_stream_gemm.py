"""The streaming GEMM of 5 to 64 rows at the edges of its blocks, stages, clusters and units, against the same sums in 64 bits
from the oracle's quantized activations.

Group sums are exact.  A warp adds at most (G / S + 7) / 8 of them with one rounding each (2^-24 of a running sum that is no
larger than the sum of the magnitudes), then come 3 additions of pairs, one per further CTA of the cluster (up to 7) and
the epilogue (2 roundings).  That bounds every output by itself; infinite scales and sums that only cancel are left out."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mllm_b200 as mb  # noqa: E402
from oracle_lib import Oracle  # noqa: E402
from test_chunk_gemm import _acts64, _weights64  # noqa: E402


def _group_magnitudes(orc, x, w64):
    """sum over K-groups of |group sum| times the row's scale, and the zero-point term's magnitude, [m, n]."""
    m, k = x.shape
    raw = np.ascontiguousarray(orc.quant_act(x)).reshape(m, -1).view(np.uint8)
    head = np.ascontiguousarray(raw[:, :8])
    recip, off = head.view(np.float32)[:, :1].astype(np.float64), head.view(np.int32)[:, 1:].astype(np.float64)
    q = raw[:, 8:8 + k].view(np.int8).astype(np.float64)
    total = np.abs(off * w64.sum(1)[None])
    for g in range(0, k, 32):
        total += np.abs(q[:, g:g + 32] @ w64[:, g:g + 32].T)
    return total * recip


def _case(m, k, ns, mode=mb.SCALE_BF16_TRUNC, odd=False, policy=mb.KERNEL_AUTO):
    orc, rng = Oracle(), np.random.default_rng(m + 7 * k + sum(ns))
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[-1], x[1] = np.abs(x[-1]) + 1, 0
    xd = torch.zeros((m, k + 3), device="cuda")  # rows that are not 16 bytes apart
    xd = (xd[:, :k] if odd else xd[:, :k].contiguous()).copy_(torch.from_numpy(x))
    a, wts = _acts64(orc, x), []
    for n in ns:
        bias = (rng.standard_normal(n) * 0.1).astype(np.float32)
        blob = mb.quant_prepack((rng.standard_normal((n, k)) * 0.02).astype(np.float32), bias, scale_mode=mode)
        wts.append((mb.W4A32Weights.from_blob(blob), *_weights64(blob, mode)))
    outs = mb.linear_forward_grouped(xd, [w for w, _, _ in wts], pdl=True, policy=policy)
    mb.check_device_status()
    rounds = ((k + 31) // 32 + 7) // 8 + 3 + 7 + 2
    for (wt, w64, bias), y in zip(wts, outs):
        want = a @ w64.T + bias
        bar = rounds * 2.0 ** -24 * (_group_magnitudes(orc, x, w64) + np.abs(bias) + np.abs(want)) + 1e-30
        assert (np.abs(y.cpu().numpy() - want) <= bar).all(), (wt.n, np.max(np.abs(y.cpu().numpy() - want) / bar))
        buf = torch.full((m, wt.n + (21 if odd else 24)), float("nan"), device="cuda")
        mb.linear_forward(xd, wt, out=buf[:, :wt.n], kernel=policy)  # the same bits by itself, and nothing outside of its columns
        mb.check_device_status()
        assert torch.equal(buf[:, :wt.n], y) and bool(torch.isnan(buf[:, wt.n:]).all())


# rows: one tile, three tiles, one and two blocks of even and uneven size; K: under a group, one partial stage, one cell in
# the second half of a stage, the border of cluster sizes 1 and 2, size 4 and 8, more stages than the ring; N: under a
# panel, one unit a cluster, several (the epilogue warps), a matrix that ends inside a later unit
@pytest.mark.parametrize("m,k,ns", [(5, 31, (33,)), (8, 1536, (1536, 40)), (9, 544, (4800,)), (17, 4448, (64, 31)), (24, 4480, (2400,)),
                                    (31, 896, (9728,)), (33, 1536, (256, 4737)), (40, 800, (64, 2500)), (41, 8960, (1536,)), (48, 1176, (1280,)),
                                    (57, 1536, (130, 7000)), (64, 10240, (2432,)), (64, 12288, (96,)), (8, 32768, (64,)), (16, 20480, (160,))])
def test_blocks_stages_and_units(m, k, ns):
    _case(m, k, ns)


@pytest.mark.parametrize("m,k,ns", [(13, 1504, (4833,)), (50, 4640, (70, 700))])
def test_fp16_scales(m, k, ns):
    _case(m, k, ns, mb.SCALE_FP16)


@pytest.mark.parametrize("m,k,ns", [(7, 1537, (129,)), (64, 1001, (4803, 31)), (20, 13000, (35,))])
def test_rows_and_outputs_off_16_bytes(m, k, ns):
    _case(m, k, ns, odd=True)


# stages of 32 K-groups: exactly one, one and a K-group, one with the second trip of a few warps, more than the ring in both
# parts of a cluster; where only 16 fit
@pytest.mark.parametrize("m,k,ns", [(8, 1024, (40,)), (16, 1056, (4801,)), (40, 608, (5000, 33)), (8, 8225, (64,)), (20, 8992, (2400,)), (56, 12288, (320,))])
def test_stages_of_32_groups(m, k, ns):
    _case(m, k, ns)


# rows that the quantization reads twice: all of them in 16-byte words with half an item at the end, and only every fourth
@pytest.mark.parametrize("m,k,ns", [(10, 12300, (65,)), (7, 12293, (33,))])
def test_long_rows(m, k, ns):
    _case(m, k, ns)


# above 64 rows, where the fastest policy takes the kernel: three to six blocks, the borders of its rows, columns and K
@pytest.mark.parametrize("m,k,ns", [(65, 1024, (31,)), (80, 1536, (1536, 256)), (97, 8960, (1536,)), (127, 4448, (4096,)), (128, 896, (896, 128, 128)),
                                    (161, 4864, (896,)), (192, 2048, (2048, 1024))])
def test_fastest_above_64_rows(m, k, ns):
    _case(m, k, ns, policy=mb.KERNEL_FASTEST)


# one tile of x where the weight tiles fill the SMs: columns of padding up to half a tile, 256 weight rows, the last panel short
@pytest.mark.parametrize("m,k,ns", [(65, 896, (8192,)), (127, 96, (4864, 4864)), (129, 512, (12900,)), (200, 224, (28672,)), (255, 1536, (8960, 8960))])
def test_fastest_tiles_of_uneven_rows(m, k, ns):
    """The fp16 tile GEMM: one truncated sum over K, K / 16 additions as in test_chunk_gemm's bar."""
    orc, rng = Oracle(), np.random.default_rng(m + k)
    x = rng.standard_normal((m, k)).astype(np.float32)
    wts = []
    for n in ns:
        blob = mb.quant_prepack((rng.standard_normal((n, k)) * 0.02).astype(np.float32))
        wts.append((mb.W4A32Weights.from_blob(blob), _weights64(blob, mb.SCALE_BF16_TRUNC)[0]))
    outs = mb.linear_forward_grouped(torch.from_numpy(x).cuda(), [w for w, _ in wts], pdl=True, policy=mb.KERNEL_FASTEST)
    mb.check_device_status()
    a = _acts64(orc, x)
    for (_, w64), y in zip(wts, outs):
        want = a @ w64.T
        assert np.linalg.norm(y.cpu().numpy() - want) <= (k / 16 / 3 + 2) * 2.0 ** -23 * np.linalg.norm(want)


@pytest.mark.parametrize("scale", [2.0 ** -120, 2.0 ** 100])
def test_far_scales(scale):
    """Group sums up to 2^15 times scales near the ends of bf16: the sixteenfold integers of the tensor cores leave no trace."""
    orc, rng = Oracle(), np.random.default_rng(3)
    m, k, n = 24, 256, 96
    nib = rng.integers(0, 256, (n, k // 2)).astype(np.uint8)
    s16 = (((rng.random((n, k // 32)) + 0.5) * scale).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    blob = mb.prepack_from_quantized(nib, s16, n, k, None, mb.SCALE_BF16_TRUNC)
    x = rng.standard_normal((m, k)).astype(np.float32)
    want = _acts64(orc, x) @ _weights64(blob, mb.SCALE_BF16_TRUNC)[0].T
    y = mb.linear_forward(torch.from_numpy(x).cuda(), mb.W4A32Weights.from_blob(blob)).cpu().numpy().astype(np.float64)
    mb.check_device_status()
    assert np.linalg.norm((y - want) / scale) <= 1e-6 * np.linalg.norm(want / scale)


@pytest.mark.parametrize("m,policy", [(24, mb.KERNEL_AUTO), (70, mb.KERNEL_AUTO), (200, mb.KERNEL_FASTEST)])
def test_halves_round_away_from_zero(m, policy):
    """Rows with range -128 .. 127 (a scale of one) or half of it and zero points at either end: every x is an integer, a half or
    next to one.  One quantum too far would be off by a hundred times the bar."""
    orc, rng = Oracle(), np.random.default_rng(m)
    k, n = 544, 64
    x = rng.integers(-256, 255, (m, k)).astype(np.float32) / 2
    x[1::4] = np.abs(x[1::4]) * np.float32(255 / 128)
    x[2::4] = -np.abs(x[2::4])
    x[3::4] = np.nextafter(x[3::4], np.float32(0) if m & 2 else np.float32(1e9), dtype=np.float32)
    x[0::2, 5], x[0::4, 7], x[0::4, 9] = 0.5, -128, 127
    blob = mb.quant_prepack((rng.standard_normal((n, k)) * 0.02).astype(np.float32))
    w64 = _weights64(blob, mb.SCALE_BF16_TRUNC)[0]
    y = mb.linear_forward(torch.from_numpy(x).cuda(), mb.W4A32Weights.from_blob(blob), kernel=policy).cpu().numpy()
    mb.check_device_status()
    bar = 40 * 2.0 ** -23 * _group_magnitudes(orc, x, w64)
    assert (np.abs(y - _acts64(orc, x) @ w64.T) <= bar).all()


def test_infinities_and_nan_in_a_row():
    """A row's infinity takes its scale to zero, a NaN counts as zero; other rows do not notice."""
    rng = np.random.default_rng(8)
    wt = mb.W4A32Weights.from_blob(mb.quant_prepack((rng.standard_normal((64, 512)) * 0.02).astype(np.float32), np.ones(64, np.float32)))
    for m, policy in ((24, mb.KERNEL_AUTO), (70, mb.KERNEL_AUTO), (200, mb.KERNEL_FASTEST)):
        x = rng.standard_normal((m, 512)).astype(np.float32)
        x[3, 17], x[5, 100] = np.inf, np.nan
        zeroed = x.copy()
        zeroed[5, 100] = 0
        run = lambda v: mb.linear_forward(torch.from_numpy(v).cuda(), wt, kernel=policy).cpu().numpy()  # noqa: E731
        got, want = run(x), run(zeroed)
        mb.check_device_status()
        rest = np.arange(m) != 3
        assert np.array_equal(got[rest], want[rest]) and np.array_equal(got[3], np.ones(64, np.float32))
