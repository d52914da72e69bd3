"""Linears called at the same time on several streams, from one host thread and from several: each call has its own activations in
operand blocks, row headers and K-split counters, so every result has the bits of the same call made alone."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import mllm_b200 as mb  # noqa: E402
from mllm_b200 import binding, w4a16  # noqa: E402

SHAPES = [(1, 1536, 1536, 0), (8, 1536, 1536, 0), (48, 1536, 1536, 0), (64, 4864, 896, 0), (96, 1536, 1536, 0), (160, 1536, 1536, 5),
          (300, 1536, 1536, 5), (513, 1536, 1536, 0)]


@pytest.fixture(scope="module")
def calls():
    """(a function of a stream, its result alone)"""
    rng, weights, out = np.random.default_rng(3), {}, []
    for m, k, n, kernel in SHAPES:
        if (k, n) not in weights:
            w = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
            weights[k, n] = mb.W4A32Weights.from_blob(mb.quant_prepack(w)), w4a16.W4A16Weights.from_blob(w4a16.quant_prepack(w))
        x = torch.randn((m, k), device="cuda")
        a, b = weights[k, n]
        out.append(lambda stream, x=x, a=a, kernel=kernel: mb.linear_forward(x, a, kernel=kernel, stream=stream))
        out.append(lambda stream, x=x, a=a: mb.linear_forward_grouped(x, [a, a], stream=stream)[1])
        out.append(lambda stream, x=x, b=b: w4a16.linear_forward(x, b, stream=stream))
    torch.cuda.synchronize()
    made = [(f, f(None)) for f in out]
    torch.cuda.synchronize()
    return made


def _wrong(calls, order, stream, own):
    """Calls in the given order on a stream (own: as the current one), then what differs."""
    got = []
    if own:
        with torch.cuda.stream(stream):
            got = [(i, calls[i][0](None)) for i in order]
    else:
        got = [(i, calls[i][0](stream)) for i in order]
    stream.synchronize()
    return [i for i, y in got if not torch.equal(y, calls[i][1])]


def test_a_captured_first_call_and_torchs_public_allocator(monkeypatch):
    """A captured call's memory is the graph's; and without torch's short way to its allocator the public one serves."""
    m, k, n = 512, 1536, 8960
    w = mb.W4A32Weights.from_blob(mb.quant_prepack((np.random.default_rng(5).standard_normal((n, k)) * 0.02).astype(np.float32)))
    x = torch.randn((m, k), device="cuda")
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        y = mb.linear_forward(x, w)
    others = [torch.full((1 << 22,), 0x7f, dtype=torch.uint8, device="cuda") for _ in range(8)]  # whatever the allocator hands out meanwhile
    y.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert all(bool((o == 0x7f).all()) for o in others)
    raw = torch._C._cuda_cudaCachingAllocator_raw_alloc  # (what the public way calls today, under whatever name)
    monkeypatch.delattr(torch._C, "_cuda_cudaCachingAllocator_raw_alloc")
    monkeypatch.setattr(torch.cuda, "caching_allocator_alloc", lambda size, device=None, stream=None: raw(size, stream))
    binding._allocator.cache_clear()
    again = mb.linear_forward(x, w), mb.linear_forward(x, w, stream=s)
    torch.cuda.synchronize()
    binding._allocator.cache_clear()
    assert torch.equal(y, again[0]) and torch.equal(y, again[1])
    mb.check_device_status()


def test_weights_loaded_on_a_stream():
    """The blob's copy belongs to the current stream, its repack to the one that is given, here one with work in front of it."""
    rng, s = np.random.default_rng(4), torch.cuda.Stream()
    for pack, load in ((mb.quant_prepack, mb.W4A32Weights), (w4a16.quant_prepack, w4a16.W4A16Weights)):
        blob = pack((rng.standard_normal((896, 1536)) * 0.02).astype(np.float32))
        with torch.cuda.stream(s):
            torch.cuda._sleep(20_000_000)
        got = load.from_blob(blob, stream=s)
        assert torch.equal(got.tiled, load.from_blob(blob).tiled)
        if load is mb.W4A32Weights:
            assert np.array_equal(got.unpack(stream=s), blob)


@pytest.mark.parametrize("own", [True, False])
def test_two_streams_in_one_thread(calls, own):
    streams, got = [torch.cuda.Stream() for _ in range(2)], []
    for i in range(40 * len(calls)):
        j, s = (7 * i) % len(calls), streams[i % 2]
        if own:
            with torch.cuda.stream(s):
                got.append((j, calls[j][0](None)))
        else:
            got.append((j, calls[j][0](s)))
    torch.cuda.synchronize()
    assert [j for j, y in got if not torch.equal(y, calls[j][1])] == []
    mb.check_device_status()


@pytest.mark.parametrize("own", [True, False])
def test_a_stream_a_thread_and_threads_on_one_stream(calls, own):
    shared, wrong = torch.cuda.Stream(), []
    jobs = []
    for t in range(4):
        order = np.random.default_rng(t).integers(0, len(calls), 200).tolist()
        stream = shared if t < 2 else torch.cuda.Stream()
        jobs.append(threading.Thread(target=lambda o=order, s=stream: wrong.append(_wrong(calls, o, s, own))))
    for j in jobs:
        j.start()
    for j in jobs:
        j.join()
    assert wrong == [[]] * 4
    mb.check_device_status()
