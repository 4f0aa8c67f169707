"""Greedy sampling: rows that do and do not start on 16 bytes, vocabularies around the 8-logit units and the slices of a row, ties, and calls on
several streams at once, which share nothing."""
import ctypes as C

import numpy as np
import pytest

from oracle.decode_step import TinyWeights

from test_decode_chain_gpu import Step
from test_decode_step_gpu import build_device_model

pytestmark = pytest.mark.gpu


def _argmax(lib, out, logits, vocab, st):
    from lmdeploy_b200 import _lib as L
    L.check(lib.b200_argmax(out.data_ptr(), logits.data_ptr(), logits.shape[0], vocab, logits.stride(0), int("bfloat" in str(logits.dtype)), st),
            "argmax")


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("vocab", [1, 7, 8, 129, 1003, 4099, 92544])
@pytest.mark.parametrize("pad", [0, 3, 8])
def test_argmax(lib, vocab, pad, dtype):
    import torch
    T, rows = getattr(torch, dtype), 33 if pad == 0 else 5                          # 33: smaller blocks
    g = torch.Generator(device="cuda").manual_seed(vocab)
    logits = torch.full((rows, vocab + pad), 100.0, dtype=T, device="cuda")         # what lies behind a row is larger than all of it
    logits[:, :vocab] = torch.randint(-20, 20, (rows, vocab), generator=g, device="cuda").to(T)        # ties all over
    logits[1, :vocab] = -float("inf")
    logits[2, vocab - 1] = 50.0
    out = torch.full((rows + 1,), -7, dtype=torch.int32, device="cuda")
    _argmax(lib, out, logits, vocab, torch.cuda.current_stream().cuda_stream)
    x = logits[:, :vocab].float().cpu().numpy()
    assert out.cpu().tolist() == [int(i) for i in x.argmax(1)] + [-7]                # numpy: the first of equal values


def test_argmax_on_two_streams(lib):
    import torch
    rows, vocab = 64, 32768
    logits = [torch.randn(rows, vocab, device="cuda", generator=torch.Generator(device="cuda").manual_seed(s)).half() for s in (1, 2)]
    refs = [x.cpu().numpy().argmax(1) for x in logits]
    outs = [torch.zeros(40, rows, dtype=torch.int32, device="cuda") for _ in logits]
    streams = [torch.cuda.Stream() for _ in logits]
    torch.cuda.synchronize()
    for i in range(40):
        for x, out, s in zip(logits, outs, streams):
            _argmax(lib, out[i], x, vocab, s.cuda_stream)
    torch.cuda.synchronize()
    for out, ref in zip(outs, refs):
        assert (out.cpu().numpy() == ref).all()


def test_steps_of_two_models_on_two_streams():
    import torch
    made = []
    for seed in (1, 2):
        w = TinyWeights(hidden=512, layers=1, heads=4, kv_heads=2, inter=1024, vocab=1024, seed=seed)
        step = Step(w, 24, 8, seed)
        made.append((build_device_model(w, 8, max_batch=32), step, step.pool(), torch.zeros(30, 24, dtype=torch.int32, device="cuda"), torch.cuda.Stream()))
    torch.cuda.synchronize()
    for i in range(30):
        for m, step, (pool, ptrs), out, s in made:
            m.decode_step(batch=24, token_ids=step.d_tok, cu_q_len=step.cu_q, cu_k_len=step.cu_k, block_ptrs=ptrs, cu_block_nums=step.cu_blocks, out_tokens=out[i],
                          max_k_len=int(step.hist.max()) + 1, stream=s)
    torch.cuda.synchronize()
    for m, step, _, out, _ in made:
        assert (out.cpu().numpy() == m.logits(24).float().cpu().numpy().argmax(1)).all()
