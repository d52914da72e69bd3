"""The head of the batched decoder: widths that end in half a step of the contraction, vocabularies that end inside a tile, rows in
one, two and three tiles of x, weights on 32 and on 16 bytes (either kind of load brings the same words, so the same bits)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
from test_decoder import SMALL, _gpu_decoder, make_model  # noqa: E402
from test_decoder_batch import FLIP_TOL, LOGIT_TOL, _rms, _run_single  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,vocab,batch", [(32, 33, 3), (96, 1, 9), (96, 4736 * 2 + 31, 17), (160, 700, 33), (128, 12000, 70)])
def test_head_of_a_batch(hidden, vocab, batch):
    import torch
    import mllm_b200 as mb
    cfg = dict(SMALL, hidden=hidden, vocab=vocab)
    w, raw = make_model(cfg, 3)
    dec = _gpu_decoder(cfg, w, raw)
    rng = np.random.default_rng(5)
    prompts = [rng.integers(0, vocab, size=int(rng.integers(1, 12))).tolist() for _ in range(batch)]
    singles = [_run_single(dec, p, 1) for p in prompts]
    emb, head = torch.from_numpy(w["embedding"]).cuda(), torch.from_numpy(w["lm_head"].astype(np.float16)).cuda()
    moved = torch.zeros(head.numel() + 16, dtype=torch.float16, device="cuda")
    moved = moved[8:8 + head.numel()].view_as(head).copy_(head)  # 16 bytes further on
    assert head.data_ptr() % 32 == 0 and moved.data_ptr() % 32 == 16
    got = []
    for table in (head, moved):
        dec.set_tables(emb, table)
        bd = mb.Qwen2BatchDecoder(dec, batch)
        for b, p in enumerate(prompts):
            bd.prefill(b, tokens=p)
        bd.decode(1)
        rows = [bd.read(b, 0, 0, want_logits=True)[2].copy() for b in range(batch)]
        for b, row in enumerate(rows):
            assert int(bd.generated(b, 1)[-1]) == int(np.argmax(row)), b
        got.append(np.stack(rows))
        mb.check_device_status()
        bd.close()
    assert np.array_equal(got[0], got[1])
    errors = [float(np.max(np.abs(row - s[2]))) / _rms(s[2]) for row, s in zip(got[0], singles)]
    assert max(errors) <= FLIP_TOL and sum(e > LOGIT_TOL for e in errors) <= max(1, batch // 10), errors
    dec.close()
