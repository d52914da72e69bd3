"""W4A16 sibling path (asymmetric int4 weights with fp32 scale/zero per group, per-block int8 activations,
fp16 output): host quantizer and CUDA path against oracle/w4a16_oracle.c.

The oracle restates mllm/Backends/Arm/Kernels/kai_linear.cpp:710-817 (weights) and the KleidiAI
activation/matmul semantics; it is NOT pinned by execution (the reference file does not compile on x86-64
and KleidiAI is absent), so the bars below are: host quantizer == oracle bit for bit; CUDA == oracle up to
the order of the fp32 additions, i.e. within 2 fp16 ulps of the value plus 1e-3 * rms of the row (dp4a
kernel); the tensor-core kernel rounds both operands once to fp16 (relative 2^-12 rms each, i.e. about
3e-4 * rms of the row after the K sum): 2 ulps plus 4e-3 * rms.
"""
import numpy as np
import pytest

from oracle_lib import Oracle, OracleW4A16


def _unpack_nibbles(q, k):
    u = np.zeros((q.shape[0], q.shape[1] * 2), np.int32)
    u[:, 0::2] = q >> 4   # even k in the high half
    u[:, 1::2] = q & 15
    return u[:, :k]


def _weights(n, k, seed, spread=0.02):
    rng = np.random.default_rng(seed)
    w = (rng.standard_normal((n, k)) * spread).astype(np.float32)
    w[0, :min(k, 32)] = 0.0               # an all-zero group
    if n > 1:
        w[1, :min(k, 32)] = np.abs(w[1, :min(k, 32)]) + 0.01   # all positive: min clamps to 0
    if n > 2:
        w[2, :min(k, 32)] = -np.abs(w[2, :min(k, 32)]) - 0.01  # all negative: max clamps to 0
    return w


# ------------------------------------------------------------------ CPU: oracle properties

@pytest.mark.parametrize("n,k", [(8, 64), (5, 100), (3, 33), (64, 1536)])
def test_oracle_weight_quantization_properties(n, k):
    """Dequantized weights are within half a step of the input, zero maps to itself, nibbles are in range."""
    o = OracleW4A16()
    w = _weights(n, k, 1)
    q, s, z, zp = o.quant_weights(w)
    nb = o.nblocks(k)
    u = _unpack_nibbles(q, k)
    se, ze = np.repeat(s, 32, 1)[:, :k], np.repeat(z, 32, 1)[:, :k]
    wd = (u - 8) * se + ze
    assert (np.abs(wd - w) <= 0.5 * se * (1 + 1e-5) + 1e-12).all()
    assert u.min() >= 0 and u.max() <= 15
    assert np.array_equal(z, (-zp.astype(np.float32)) * s)       # the rescale of kai_linear.cpp:797-805
    # an all-zero group: scale 1 and, by the reference's comparison (8 < 7 is false), zero point 7, nibble 15
    assert (s[0, 0], zp[0, 0]) == (1.0, 7) and (u[0, :min(k, 32)] == 15).all() and z[0, 0] == -7.0
    if n > 2:
        assert zp[1, 0] == -8 and zp[2, 0] == 7                  # one-sided groups use the whole range
    assert s.shape == (n, nb)


def test_oracle_activation_quantization_properties():
    o = OracleW4A16()
    rng = np.random.default_rng(2)
    x = rng.standard_normal((4, 100)).astype(np.float32) * 3
    x[1, :32] = 0
    a_q, a_s = o.quant_act(x)
    assert a_q.shape == (4, 128) and (a_q[:, 100:] == 0).all()
    assert (np.abs(a_q) <= 127).all() and a_s[1, 0] == 0 and (a_q[1, :32] == 0).all()
    xd = a_q[:, :100] * np.repeat(a_s, 32, 1)[:, :100]
    assert (np.abs(xd - x) <= 0.5 * np.repeat(a_s, 32, 1)[:, :100] * (1 + 1e-5)).all()
    # the largest element of every block maps to +-127
    blk = np.abs(a_q.reshape(4, 4, 32)).max(-1)
    assert (blk[a_s > 0] == 127).all()


def test_oracle_on_the_reference_fixture():
    """Inputs of KaiLinear_f16_qsi8d32p_qai4c32p_mxk_nxk_Test (tests/Arm/KaiLinearTest.hpp:479-594): M=32,
    K=N=64, srand 4568/4572/4576.  The fixture's own check (1e-2 relative to a dense fp16 product) is beyond
    any 4-bit quantizer on these inputs (uniform [-1,1] weights: step 2/15, expected error ~7 % of an output's
    typical size), so what is asserted here is the error that int4 + int8 quantization predicts."""
    o, o32 = OracleW4A16(), Oracle()
    m, k, n = 32, 64, 64
    x = o.fill_uniform_random_f16(m * k, 4568).reshape(m, k)
    w = o32.fill_uniform_random(n * k, 4572).reshape(n, k)
    b = o32.fill_uniform_random(n, 4576)
    assert x.dtype == np.float16 and abs(float(x.astype(np.float32).mean())) < 0.05
    q, s, z, _ = o.quant_weights(w)
    y = o.linear(x, q, s, z, b).astype(np.float64)
    dense = x.astype(np.float64) @ w.astype(np.float64).T + b
    err = y - dense
    # weight error uniform in +-step/2 (sigma = step/sqrt(12)), |x| rms = 1/sqrt(3), K = 64 terms
    predicted = (2 / 15) / np.sqrt(12) * (1 / np.sqrt(3)) * np.sqrt(k)
    assert 0.6 * predicted < err.std() < 1.4 * predicted
    assert abs(err.mean()) < 0.1 * predicted


def test_oracle_matmul_equals_dequantized_product():
    """The block formula equals the plain product of the dequantized operands."""
    o = OracleW4A16()
    rng = np.random.default_rng(3)
    m, k, n = 3, 96, 7
    x = rng.standard_normal((m, k)).astype(np.float32)
    w = _weights(n, k, 4, spread=0.5)
    b = rng.standard_normal(n).astype(np.float32)
    q, s, z, _ = o.quant_weights(w)
    a_q, a_s = o.quant_act(x)
    y = o.linear(x, q, s, z, b).astype(np.float64)
    wd = (_unpack_nibbles(q, k) - 8) * np.repeat(s, 32, 1).astype(np.float64) + np.repeat(z, 32, 1)
    xd = a_q[:, :k].astype(np.float64) * np.repeat(a_s, 32, 1)
    ref = xd @ wd.T + b
    assert np.abs(y - ref).max() <= 2e-3 * np.abs(ref).max()   # fp16 output rounding


# ------------------------------------------------------------------ CPU: host quantizer == oracle

@pytest.mark.parametrize("n,k,has_bias", [(8, 64, True), (5, 100, False), (3, 33, True), (96, 1536, True),
                                          (33, 1176, False)])
def test_host_quantizer_matches_oracle_bit_for_bit(n, k, has_bias):
    from mllm_b200 import w4a16
    o = OracleW4A16()
    w = _weights(n, k, 10 + n)
    bias = np.random.default_rng(5).standard_normal(n).astype(np.float32) if has_bias else None
    blob = w4a16.quant_prepack(w, bias)
    assert w4a16.blob_info(blob) == (n, k, int(has_bias))
    nib, sc, zr, bs = w4a16.blob_sections(blob)
    q, s, z, _ = o.quant_weights(w)
    assert np.array_equal(nib, q)
    assert np.array_equal(sc.view(np.uint32), s.view(np.uint32))
    assert np.array_equal(zr.view(np.uint32), z.view(np.uint32))
    if has_bias:
        assert np.array_equal(bs, bias)
    else:
        assert bs is None


def test_host_abi_argument_checks():
    import ctypes as C
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    L = mb.lib()
    out = C.c_size_t()
    assert L.mllmb200_w4a16_prepack_size(0, 64, 0, C.byref(out)) == 1
    assert L.mllmb200_w4a16_prepack_size(8, 64, 0, None) == 1
    assert L.mllmb200_w4a16_tiled_size(8, 0, C.byref(out)) == 1
    assert L.mllmb200_w4a16_workspace_size(1, 64, 0, C.byref(out)) == 1
    assert L.mllmb200_w4a16_linear_forward(None, 0, None, None, None, 1, 64, 8, 64, 8, None) == 1
    blob = w4a16.quant_prepack(np.ones((8, 64), np.float32))
    w32 = mb.quant_prepack(np.ones((8, 64), np.float32))
    with pytest.raises(mb.MllmB200Error):
        w4a16.blob_info(w32)          # a W4A32 blob is not a W4A16 blob ...
    with pytest.raises(mb.MllmB200Error):
        mb.blob_info(blob)            # ... and the other way round
    # sizes: 8 rows x (32 nibble bytes + 2 groups x 8 bytes) + header
    assert w4a16.prepack_size(8, 64, False) == 64 + 8 * 32 + 8 * 2 * 4 * 2
    assert w4a16.tiled_size(8, 64) == 256 + 2 * 768 + 256   # header, 1 panel x 2 groups, bias rounded to 256


# ------------------------------------------------------------------ GPU parity

def _bar(y_ref, tensor_path=False):
    y = y_ref.astype(np.float32)
    rms = np.sqrt((y.astype(np.float64) ** 2).mean(axis=1, keepdims=True)).astype(np.float32)
    return 2 * np.spacing(np.abs(y_ref)).astype(np.float32) + (4e-3 if tensor_path else 1e-3) * rms


def _auto_is_tensor(m, n):
    """The library's automatic choice (launch_w4a16_linear): tensor cores for large M, or mid M on wide matrices."""
    return m >= 128 or (m >= 32 and n >= 8192)


SHAPES = [
    (1, 1536, 1536), (1, 1536, 256), (1, 1536, 8960), (1, 8960, 1536),   # the decoder's linears at M = 1
    (2, 64, 64), (3, 100, 33), (4, 33, 5), (7, 1176, 96), (16, 256, 40),
    (32, 64, 64),                                                          # the reference fixture's shape
    (40, 1536, 256), (130, 512, 320), (512, 1536, 256),
]
# (m, k, n, kernel): the tensor-core kernel on every tile width, ragged M / N / K, and the dp4a kernel at large M
TENSOR_SHAPES = [
    (64, 256, 128, 4), (100, 100, 33, 4), (130, 512, 320, 4), (200, 1176, 1280, 4), (512, 1536, 1536, 4),
    (512, 1536, 8960, 4), (512, 8960, 1536, 4), (300, 1536, 8960, 0), (70, 256, 96, 0), (512, 1536, 256, 2), (130, 512, 320, 2), (63, 8192, 512, 0), (40, 256, 8200, 0), (16, 512, 96, 4),
    (1, 1536, 256, 2), (3, 100, 33, 2), (4, 8960, 1536, 2),   # the record-based dp4a kernel where auto takes the fused one
    # one tile of x as wide as the rows need where the weight tiles fill the SMs, on both sides of its limits in rows and weight rows
    (65, 96, 8065, 4), (127, 512, 8200, 4), (64, 96, 8200, 4), (100, 96, 8064, 4), (129, 224, 12673, 4), (255, 96, 12800, 4), (140, 96, 12672, 4),
]


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n,kernel", TENSOR_SHAPES)
def test_gpu_tensor_core_kernel_matches_oracle(m, k, n, kernel):
    import torch
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    o = OracleW4A16()
    rng = np.random.default_rng(m + k + n)
    w = _weights(n, k, m + n + 1)
    bias = (rng.standard_normal(n) * 0.1).astype(np.float32) if n % 2 == 0 else None
    x = rng.standard_normal((m, k)).astype(np.float16 if (m + k) % 3 == 0 else np.float32)
    blob = w4a16.quant_prepack(w, bias)
    nib, sc, zr, _ = w4a16.blob_sections(blob)
    ref = o.linear(x, nib.copy(), sc.copy(), zr.copy(), bias)
    y = w4a16.linear_forward(torch.from_numpy(x).cuda(), w4a16.W4A16Weights.from_blob(blob), kernel=kernel)
    torch.cuda.synchronize()
    mb.check_device_status()
    got = y.cpu().numpy()
    tensor = kernel == 4 or (kernel == 0 and _auto_is_tensor(m, n))
    diff = np.abs(got.astype(np.float32) - ref.astype(np.float32))
    assert (diff <= _bar(ref, tensor)).all(), f"max diff {diff.max()} at {np.unravel_index(diff.argmax(), diff.shape)}"
    rms = np.sqrt((ref.astype(np.float64) ** 2).mean())
    print(f"m={m} k={k} n={n} kernel={kernel}: rms err / rms y = {np.sqrt((diff.astype(np.float64) ** 2).mean()) / rms:.2e}, "
          f"identical fp16 outputs {(got == ref).mean():.3f}")
    assert np.sqrt((diff.astype(np.float64) ** 2).mean()) <= (8e-4 if tensor else 4e-4) * rms


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,n", SHAPES)
@pytest.mark.parametrize("x_dtype", ["f32", "f16"])
def test_gpu_linear_matches_oracle(m, k, n, x_dtype):
    import torch
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    o = OracleW4A16()
    rng = np.random.default_rng(m * 7 + k + n)
    w = _weights(n, k, m + n)
    bias = (rng.standard_normal(n) * 0.1).astype(np.float32) if (m + n) % 2 == 0 else None
    x = rng.standard_normal((m, k)).astype(np.float32)
    x[0, :min(k, 32)] = 0.0    # an all-zero activation block: scale 0
    if x_dtype == "f16":
        x = x.astype(np.float16)
    blob = w4a16.quant_prepack(w, bias)
    nib, sc, zr, _ = w4a16.blob_sections(blob)
    ref = o.linear(x, nib.copy(), sc.copy(), zr.copy(), bias)
    wts = w4a16.W4A16Weights.from_blob(blob)
    xt = torch.from_numpy(x).cuda()
    y = w4a16.linear_forward(xt, wts)
    torch.cuda.synchronize()
    mb.check_device_status()
    got = y.cpu().numpy()
    assert got.dtype == np.float16 and got.shape == (m, n)
    diff = np.abs(got.astype(np.float32) - ref.astype(np.float32))
    tensor = _auto_is_tensor(m, n)   # the automatic choice
    assert (diff <= _bar(ref, tensor)).all(), f"max diff {diff.max()} at {np.unravel_index(diff.argmax(), diff.shape)}"
    # most outputs are the same fp16 value
    assert (got == ref).mean() > (0.3 if tensor else 0.9)


@pytest.mark.gpu
def test_gpu_reference_fixture():
    """The reference fixture's inputs (fp16 activations) through the CUDA path == oracle."""
    import torch
    from mllm_b200 import w4a16
    o, o32 = OracleW4A16(), Oracle()
    m, k, n = 32, 64, 64
    x = o.fill_uniform_random_f16(m * k, 4568).reshape(m, k)
    w = o32.fill_uniform_random(n * k, 4572).reshape(n, k)
    b = o32.fill_uniform_random(n, 4576)
    blob = w4a16.quant_prepack(w, b)
    nib, sc, zr, _ = w4a16.blob_sections(blob)
    ref = o.linear(x, nib.copy(), sc.copy(), zr.copy(), b)
    y = w4a16.linear_forward(torch.from_numpy(x).cuda(), w4a16.W4A16Weights.from_blob(blob)).cpu().numpy()
    assert (np.abs(y.astype(np.float32) - ref.astype(np.float32)) <= _bar(ref)).all()


@pytest.mark.gpu
def test_gpu_row_shards_equal_the_whole():
    """Output-channel shards (tensor parallel) reproduce the matching columns of the unsharded result."""
    import torch
    from mllm_b200 import w4a16
    rng = np.random.default_rng(11)
    m, k, n = 5, 512, 320
    w = _weights(n, k, 12)
    bias = rng.standard_normal(n).astype(np.float32)
    blob = w4a16.quant_prepack(w, bias)
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).cuda()
    full = w4a16.linear_forward(x, w4a16.W4A16Weights.from_blob(blob)).cpu().numpy()
    for g in (2, 5):
        per = n // g
        parts = [w4a16.linear_forward(x, w4a16.W4A16Weights.from_blob(blob, row_begin=r * per, row_count=per))
                 .cpu().numpy() for r in range(g)]
        assert np.array_equal(np.concatenate(parts, axis=1), full)


@pytest.mark.gpu
def test_gpu_strided_rows_and_bad_header():
    import torch
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    rng = np.random.default_rng(13)
    m, k, n = 6, 96, 40
    blob = w4a16.quant_prepack(_weights(n, k, 14))
    wts = w4a16.W4A16Weights.from_blob(blob)
    xs = torch.from_numpy(rng.standard_normal((m, k + 9)).astype(np.float32)).cuda()
    ys = torch.zeros((m, n + 3), dtype=torch.float16, device="cuda")
    dense = w4a16.linear_forward(xs[:, :k].contiguous(), wts)
    w4a16.linear_forward(xs[:, :k], wts, out=ys[:, :n])
    assert torch.equal(ys[:, :n], dense) and (ys[:, n:] == 0).all()
    # a W4A32 tile buffer handed to the W4A16 entry point is refused through the device status word
    w32 = mb.W4A32Weights.from_blob(mb.quant_prepack(np.ones((n, k), np.float32)))
    fake = w4a16.W4A16Weights(w32.tiled, n, k, 0)
    w4a16.linear_forward(xs[:, :k].contiguous(), fake)
    torch.cuda.synchronize()
    with pytest.raises(mb.MllmB200Error):
        mb.check_device_status()
    mb.check_device_status()   # the status word is cleared by the read


@pytest.mark.gpu
def test_gpu_chain_with_programmatic_dependent_launch():
    """A chain of single-launch linears (each reads what the previous one wrote) gives the same bits with and
    without programmatic dependent launch."""
    import torch
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    rng = np.random.default_rng(21)
    dims = [1536, 256, 1536, 512, 1536]
    wts = [w4a16.W4A16Weights.from_blob(w4a16.quant_prepack(_weights(dims[i + 1], dims[i], 30 + i, spread=0.05)))
           for i in range(len(dims) - 1)]
    x0 = torch.from_numpy(rng.standard_normal((1, dims[0])).astype(np.float16)).cuda()
    outs = {}
    for pdl in (False, True):
        bufs = [torch.zeros((1, d), dtype=torch.float16, device="cuda") for d in dims[1:]]
        for _ in range(3):   # repeated so that a kernel could overtake the one before it if the ordering were wrong
            cur = x0
            for w, b in zip(wts, bufs):
                w4a16.linear_forward(cur, w, out=b, pdl=pdl)
                cur = b
        torch.cuda.synchronize()
        mb.check_device_status()
        outs[pdl] = [b.cpu().numpy() for b in bufs]
    for a, b in zip(outs[False], outs[True]):
        assert np.array_equal(a, b)
    assert np.abs(outs[True][-1].astype(np.float32)).max() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("m,k,ns", [(1, 1536, (1536, 256, 256)), (1, 1536, (8960, 8960)), (3, 100, (33, 5, 64, 40)),
                                    (4, 1536, (8960, 8960)), (40, 256, (96, 64)), (130, 512, (320, 64)),
                                    (40, 256, (4200, 4100)), (512, 1536, (1536, 256, 256))])
def test_gpu_grouped_calls_match_oracle(m, k, ns):
    """q/k/v- and gate/up-style groups: one launch at small M, per-matrix forwards otherwise; each output
    against the oracle, and (same kernels, same order of additions within a matrix's own launch or not) within
    the bar of the single calls."""
    import torch
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    o = OracleW4A16()
    rng = np.random.default_rng(m + k + sum(ns))
    x = rng.standard_normal((m, k)).astype(np.float16)
    blobs = [w4a16.quant_prepack(_weights(n, k, 50 + i), (rng.standard_normal(n) * 0.1).astype(np.float32) if i % 2 == 0 else None)
             for i, n in enumerate(ns)]
    wts = [w4a16.W4A16Weights.from_blob(b) for b in blobs]
    outs = w4a16.linear_forward_grouped(torch.from_numpy(x).cuda(), wts, pdl=True)
    torch.cuda.synchronize()
    mb.check_device_status()
    for blob, y in zip(blobs, outs):
        nib, sc, zr, bias = w4a16.blob_sections(blob)
        ref = o.linear(x, nib.copy(), sc.copy(), zr.copy(), None if bias is None else bias.copy())
        diff = np.abs(y.cpu().numpy().astype(np.float32) - ref.astype(np.float32))
        assert (diff <= _bar(ref, _auto_is_tensor(m, sum(ns)))).all(), f"max diff {diff.max()}"   # the group decides as a whole


@pytest.mark.gpu
def test_gpu_full_size_matrix():
    """BASELINE config 4's matrix (28672 x 8192): M = 2 against the oracle (records + dp4a path: the matrix is past
    the single-launch kernel's size rule), and at M = 2048 the tensor-core kernel against the dp4a kernel on the
    same inputs (the oracle would need minutes there); 8 row shards reproduce the whole within the same bar."""
    import torch
    from mllm_b200 import w4a16
    import mllm_b200 as mb
    o = OracleW4A16()
    n, k = 28672, 8192
    rng = np.random.default_rng(77)
    w = (rng.standard_normal((n, k), dtype=np.float32) * 0.02)
    blob = w4a16.quant_prepack(w)
    del w
    nib, sc, zr, _ = w4a16.blob_sections(blob)
    wts = w4a16.W4A16Weights.from_blob(blob)
    x2 = rng.standard_normal((2, k)).astype(np.float16)
    ref = o.linear(x2, nib.copy(), sc.copy(), zr.copy())
    y2 = w4a16.linear_forward(torch.from_numpy(x2).cuda(), wts)
    torch.cuda.synchronize()
    mb.check_device_status()
    diff = np.abs(y2.cpu().numpy().astype(np.float32) - ref.astype(np.float32))
    assert (diff <= _bar(ref)).all(), f"max diff {diff.max()}"
    # shards
    per = n // 8
    parts = [w4a16.linear_forward(torch.from_numpy(x2).cuda(),
                                  w4a16.W4A16Weights.from_blob(blob, row_begin=r * per, row_count=per)) for r in range(8)]
    # a shard has 112 row panels and splits K over three slices where the whole matrix (896 panels) uses one:
    # the fp32 additions are ordered differently, so the shards match within the dp4a bar, not bit for bit
    got = torch.cat(parts, dim=1).cpu().numpy()
    diff = np.abs(got.astype(np.float32) - ref.astype(np.float32))
    assert (diff <= _bar(ref)).all(), f"shards: max diff {diff.max()}"
    assert (got == y2.cpu().numpy()).mean() > 0.99
    # tensor-core kernel vs the exact dp4a kernel at the bench's M
    xm = torch.from_numpy(rng.standard_normal((2048, k)).astype(np.float16)).cuda()
    y_tc = w4a16.linear_forward(xm, wts)                       # auto: tensor cores
    y_dp = w4a16.linear_forward(xm, wts, kernel=w4a16.KERNEL_DP4A)
    torch.cuda.synchronize()
    mb.check_device_status()
    a, b = y_tc.float(), y_dp.float()
    rms = b.pow(2).mean(dim=1, keepdim=True).sqrt()
    ulp = torch.from_numpy(np.spacing(np.abs(y_dp.cpu().numpy())).astype(np.float32)).cuda()
    assert bool(((a - b).abs() <= 2 * ulp + 4e-3 * rms).all())
    assert float((a - b).pow(2).mean().sqrt() / b.pow(2).mean().sqrt()) < 8e-4
