"""A decode step against its parts: b200_model_decode_step has the bits of the public operators called one after another on packed
activations, whatever the number of rows (a linear layer's sums run in one order, so the cache's bytes do not depend on which kernel a
layer of few tokens would otherwise get).  And a step of more rows than the small models of test_decode_step_gpu have against the oracle."""
import ctypes as C

import numpy as np
import pytest

from oracle import attention as OA
from oracle.decode_step import TinyWeights, decode_step
from oracle.numerics import F16

from harness import from_dev_T
from test_decode_step_gpu import build_device_model

pytestmark = pytest.mark.gpu

ROPE = OA.RopeParam(type=OA.ROPE_DEFAULT, dim=128, base=1e4)


class Step:
    def __init__(self, w, rows, kv_bits, seed=0):
        import torch
        rng = np.random.default_rng(seed)
        self.w, self.B, self.kv_bits = w, rows, kv_bits
        self.hist = np.array([i * 37 % 131 for i in range(rows)], np.int32)
        counts = [(int(h) + 1 + 63) // 64 for h in self.hist]
        self.cache = OA.PagedKvCache(sum(counts) + 2, w.layers, OA.KvLayout(w.kv_heads, 64, 128, kv_bits), F16)
        perm, o, self.tables = rng.permutation(sum(counts) + 2), 0, []
        for n in counts:
            self.tables.append(perm[o:o + n].tolist())
            o += n
        for l in range(w.layers):
            for b, h in enumerate(self.hist):
                if h:
                    k, v = (OA.rn(rng.standard_normal((int(h), w.kv_heads, 128)).astype(np.float32), F16) for _ in range(2))
                    OA.process_kv(self.cache, self.tables[b], l, 0, k, v, ROPE)
        self.tokens = rng.integers(0, w.vocab, rows).astype(np.int32)
        self.cu_blocks = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device="cuda")
        self.cu_q = torch.arange(rows + 1, dtype=torch.int32, device="cuda")
        self.cu_k = torch.tensor(np.concatenate([[0], np.cumsum(self.hist + 1)]), dtype=torch.int32, device="cuda")
        self.d_tok = torch.from_numpy(self.tokens).cuda()
        self.policy = 0 if kv_bits == 16 else kv_bits

    def pool(self):
        import torch
        pool = torch.from_numpy(self.cache.pool.copy()).cuda()
        ptrs = torch.tensor([pool.data_ptr() + int(b) * self.cache.block_bytes for t in self.tables for b in t], dtype=torch.int64, device="cuda")
        return pool, ptrs

    def whole(self, m):
        import torch
        pool, ptrs = self.pool()
        out = torch.zeros(self.B, dtype=torch.int32, device="cuda")
        m.decode_step(batch=self.B, token_ids=self.d_tok, cu_q_len=self.cu_q, cu_k_len=self.cu_k, block_ptrs=ptrs, cu_block_nums=self.cu_blocks, out_tokens=out,
                      max_k_len=int(self.hist.max()) + 1)
        torch.cuda.synchronize()
        return m.logits(self.B).clone(), pool, out

    def chain(self, m, lib):
        import torch
        from lmdeploy_b200 import _lib as L
        from lmdeploy_b200.turbomind.runtime import PreparedLinear
        w, B, T, st = self.w, self.B, torch.float16, torch.cuda.current_stream().cuda_stream
        lin = [k for k in m._keep if isinstance(k, PreparedLinear)]
        embed, final_norm, *norms = [k for k in m._keep if not isinstance(k, PreparedLinear)]
        mt, H, D = (B + 15) // 16 * 16, w.hidden, 128
        qkv_dim = (w.heads + 2 * w.kv_heads) * D
        def buf(n): return torch.zeros(mt, n, dtype=T, device="cuda")
        residual, xp, qkv, attn, o, act, logits = buf(H), buf(H), buf(qkv_dim), buf(w.heads * D), buf(H), buf(w.inter), buf(m.vocab_local)
        ws = torch.zeros(max(lib.b200_linear_workspace_bytes(C.byref(x.desc), mt) for x in lin), dtype=torch.uint8, device="cuda")

        def linear(x, src, dst, ldy, epilogue=0, out_mt=0):
            L.check(lib.b200_linear_forward_packed(C.byref(x.desc), src.data_ptr(), mt, B, dst.data_ptr(), ldy, epilogue, out_mt, ws.data_ptr(), ws.numel(), st), "packed")

        def norm(weight):
            L.check(lib.b200_residual_rmsnorm(xp.data_ptr(), mt, residual.data_ptr(), o.data_ptr(), weight.data_ptr(), None, B, H, m.cfg.norm_eps, 0, st), "norm")

        pool, ptrs = self.pool()
        p = L.AttentionParams()
        p.out, p.q, p.stride, p.out_packed_mt = attn.data_ptr(), qkv.data_ptr(), qkv_dim, mt
        p.k, p.v = p.q + 2 * w.heads * D, p.q + 2 * (w.heads + w.kv_heads) * D
        p.cu_q_len, p.cu_k_len, p.block_ptrs, p.cu_block_nums = (t.data_ptr() for t in (self.cu_q, self.cu_k, ptrs, self.cu_blocks))
        p.block_len, p.token_num, p.batch_size, p.max_k_len = 64, B, B, int(self.hist.max()) + 1
        p.num_heads, p.num_kv_heads, p.size_per_head, p.inv_sqrt_dh = w.heads, w.kv_heads, D, m.cfg.inv_sqrt_dh
        p.rope, p.quant_policy, p.dtype = m.cfg.rope, self.policy, 0
        plan, table = torch.zeros(B + 1, dtype=torch.int32, device="cuda"), torch.zeros(B, D, dtype=torch.float32, device="cuda")
        aws = torch.zeros(lib.b200_decode_attention_workspace_bytes(B, w.heads, w.kv_heads), dtype=torch.uint8, device="cuda")
        p.workspace, p.workspace_bytes, p.plan, p.rope_table, p.stream = aws.data_ptr(), aws.numel(), plan.data_ptr(), table.data_ptr(), st
        L.check(lib.b200_embedding_lookup(residual.data_ptr(), embed.data_ptr(), self.d_tok.data_ptr(), B, H, w.vocab, 0, st), "embedding")
        L.check(lib.b200_rmsnorm(xp.data_ptr(), mt, residual.data_ptr(), norms[0].data_ptr(), B, H, m.cfg.norm_eps, 0, st), "rmsnorm")
        L.check(lib.b200_decode_attention_plan(plan.data_ptr(), p.cu_k_len, None, B, st), "plan")
        L.check(lib.b200_rope_table(table.data_ptr(), C.byref(p.rope), p.cu_q_len, p.cu_k_len, B, B, st), "rope")
        for l in range(w.layers):
            w_qkv, wo, w13, w2 = lin[4 * l:4 * l + 4]
            linear(w_qkv, xp, qkv, qkv_dim)
            p.layer_offset = l * m.layer_bytes
            L.check(lib.b200_decode_attention(C.byref(p)), "attention")
            linear(wo, attn, o, H)
            norm(norms[2 * l + 1])
            linear(w13, xp, act, w.inter, 1, mt)
            linear(w2, act, o, H)
            norm(norms[2 * l + 2] if l + 1 < w.layers else final_norm)
        linear(lin[-1], xp, logits, m.vocab_local)
        torch.cuda.synchronize()
        return logits[:B], pool


@pytest.mark.parametrize("rows", [1, 5, 17, 24, 25, 40])
@pytest.mark.parametrize("fmt,kv_bits", [("awq", 8), ("fp8", 4), ("fp16", 16)])
def test_step_has_the_bits_of_its_packed_operators(lib, fmt, kv_bits, rows):
    w = TinyWeights(hidden=512, layers=2, heads=4, kv_heads=2, inter=1024, vocab=1024, fmt=fmt, seed=rows)
    step = Step(w, rows, kv_bits)
    m = build_device_model(w, step.policy, max_batch=64)
    logits, pool, tokens = step.whole(m)
    ref, ref_pool = step.chain(m, lib)
    assert (logits == ref).all() and (pool == ref_pool).all()
    assert (tokens.long() == ref.float().argmax(-1)).all()


@pytest.mark.parametrize("fmt,kv_bits", [("awq", 8), ("fp8", 8), ("fp16", 4)])
@pytest.mark.parametrize("rows", [25, 40, 64])
def test_step_of_more_rows_matches_the_oracle(fmt, kv_bits, rows):
    """Bars of test_decode_step_gpu: three chained f16 products per layer, bytes of deeper layers may fall to the neighbouring code."""
    w = TinyWeights(hidden=512, layers=2, heads=4, kv_heads=2, inter=1024, vocab=1024, fmt=fmt, seed=rows)
    step = Step(w, rows, kv_bits, seed=1)
    logits, pool, _ = step.whole(build_device_model(w, step.policy, max_batch=64))
    ref, _ = decode_step(w, step.tokens, step.cache, step.tables, step.hist, ROPE)
    assert (pool.cpu().numpy() == step.cache.pool).mean() > 0.999
    assert np.abs(from_dev_T(logits, F16) - ref).max() <= 4e-3
