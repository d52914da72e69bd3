"""The engine's norms with an input convolution: many rows a step (shared memory's rows, shares of one and two tokens, the rows in front
of a block recomputed) and one token a sequence, over taps and widths at the edges of what a thread and a warp hold."""
import os
import sys
import threading

import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import lm_models as M  # noqa: E402
import vupuzen_oracle as V  # noqa: E402
from lm_case import Case  # noqa: E402


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,taps", [(72, 4), (1024, 2), (1032, 3), (1536, 4), (2048, 3), (2056, 4), (2560, 1)])
def test_convolution_in_steps(width, taps, dtype, tmp_path):
    cfg = M.config(width, 120, [M.layer("attention", M.attention(2, 1, 32, 32, 25), 64), M.layer("attention", M.attention(2, 2, 32, 16, 30))], taps=taps)
    w = M.weights(cfg, 5)
    c = Case(M.write(tmp_path / "m", cfg, w), V, cfg, w, dtype, max_seqs=6, max_ctx=400, max_rows=720)
    toks = [c.tokens(400, seed=i) for i in range(6)]
    want = [c.oracle(t) for t in toks]
    at, slots = [0] * 6, [c.model.acquire() for _ in toks]
    got = [[] for _ in toks]
    # shares of a step: many rows (and a new sequence of one), short ones in front of and behind long ones, decode, and so on
    for counts in ([1, 300, 2, 1, 60, 3], [1] * 6, [1] * 6, [1, 1, 330, 2, 1, 13], [1] * 6, [31, 7, 1, 300, 1, 300], [1] * 6):
        part = [(s, t[a:a + n]) for s, t, a, n in zip(slots, toks, at, counts)]
        rows = c.model.step(part, list(range(sum(counts))))
        for i, n in enumerate(counts):
            got[i].append(rows[sum(counts[:i]):sum(counts[:i + 1])])
            at[i] += n
    c.model.check_device_status()
    for g, o, a in zip(got, want, at):
        c.check(np.concatenate(g), o[:a])
    c.model.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,taps", [(1536, 1), (2048, 1), (2056, 4), (2304, 2), (4096, 3)])
def test_many_rows_of_wide_models(width, taps, dtype, tmp_path):
    """Above 2048 columns a block makes passes of 8 rows and keeps three: 18 rows and more a block, sequences that begin and end in every
    place of a pass, rows in front of a block from the sequence before.  Without a convolution: more rows than one wave of the larger blocks."""
    cfg = M.config(width, 60, [M.layer("attention", M.attention(1, 1, 16, 16, 25), 64)], taps=taps)
    w = M.weights(cfg, 5)
    c = Case(M.write(tmp_path / "m", cfg, w), V, cfg, w, dtype, max_seqs=7, max_ctx=1500, max_rows=2500)
    steps = [[1, 1100, 2, 700, 3, 400, 260], [1, 1, 200, 500, 1, 900, 740]]
    toks = [c.tokens(sum(s[i] for s in steps), seed=i) for i in range(7)]
    want = [c.oracle(t) for t in toks]
    at, slots = [0] * 7, [c.model.acquire() for _ in toks]
    for counts in steps:
        rows = c.model.step([(s, t[a:a + n]) for s, t, a, n in zip(slots, toks, at, counts)], list(range(sum(counts))))
        c.model.check_device_status()
        for i, n in enumerate(counts):
            c.check(rows[sum(counts[:i]):sum(counts[:i + 1])], want[i][at[i]:at[i] + n])
            at[i] += n
    c.model.close()


def test_engines_of_two_widths_in_two_threads(tmp_path):
    """Widths that share the kernels of the norms but not the shared memory these ask for: neither engine's launches may set a limit
    that the other's, from another host thread, then exceed."""
    cases = []
    for width in (1152, 1536):  # many rows: one instance; and one instance of the kernel for many taps
        for taps in (4, 12):
            cfg = M.config(width, 60, [M.layer("attention", M.attention(1, 1, 16, 16, 25))] * 4, taps=taps)
            c = Case(M.write(tmp_path / f"{width}_{taps}", cfg, M.weights(cfg, 5)), V, cfg, None, "bfloat16", max_seqs=1, max_ctx=320, max_rows=320)
            toks = c.tokens(300)
            cases.append((c, toks, c.run(toks)))
    errors = []

    def step(c, toks, want):
        try:
            for _ in range(150):
                slot = c.model.acquire()
                got = c.model.step([(slot, toks)], list(range(len(toks))))
                c.model.release(slot)
                np.testing.assert_array_equal(got, want)
        except Exception as e:
            errors.append(e)
    jobs = [threading.Thread(target=step, args=a) for a in cases]
    for j in jobs:
        j.start()
    for j in jobs:
        j.join()
    for c, _, _ in cases:
        c.model.close()
    assert not errors, errors[0]
