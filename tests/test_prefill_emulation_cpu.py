"""The arithmetic and the operand addresses of csrc/prefill_attention.cuh, followed on the CPU and checked against the independent oracle.

Units of two tiles of 128 rows (row -> (token, head) stacking), page addressing (data and parameter regions, int4 nibble order) by the loaders' map of
16-byte units, the operand tiles' byte addresses (Q [d/8][row][8]; K and V alike [d/8][key][8]: K-major operand of Q.K^T, MN-major operand of P.V), key
tiles of 128 per tile of rows, causal mask, dead-key zeroing, online softmax, and the partials of a piece whose keys lie in several ranges, combined in
order.  The tcgen05.mma groups are replaced by readers of the UMMA canonical layouts (no swizzle; tools/umma_probe.cu verified them on hardware) followed
by a float64 matmul.  How the ranges are cut is checked on the kernels' own code in test_prefill_work_cpu.py."""
import numpy as np
import pytest

from oracle import attention as OA
from oracle.numerics import F16, from_bits, rn, to_bits

ROWS, KEYS, D, LOADERS, START = 128, 128, 128, 7, 2


def read_operand(buf, rows, ks, lbo, sbo):
    """UMMA canonical K-major, no swizzle: -> float32 [rows, ks] from a uint8 buffer."""
    r = np.arange(rows)[:, None]
    k = np.arange(ks)[None, :]
    return _halves(buf, (k // 8) * lbo + (r // 8) * sbo + (r % 8) * 16 + (k % 8) * 2)


def read_mn_major(buf, n, ks, k_stride, n_stride):
    """UMMA canonical MN-major, no swizzle: 8 x 8 blocks, a row of 8 n-values per k; blocks k_stride / n_stride bytes apart -> float32 [ks, n]."""
    k = np.arange(ks)[:, None]
    c = np.arange(n)[None, :]
    return _halves(buf, (c // 8) * n_stride + (k // 8) * k_stride + (k % 8) * 16 + (c % 8) * 2)


def _halves(buf, addr):
    return from_bits(buf[addr].astype(np.uint16) | (buf[addr + 1].astype(np.uint16) << 8), F16)


def put16(buf, addr, halves):
    """st.shared.v4.b32: 8 T values (as float32 exact in T) at byte address addr."""
    b = to_bits(np.asarray(halves, np.float32), F16).astype(np.uint16)
    buf[addr:addr + 16:2] = b & 0xFF
    buf[addr + 1:addr + 16:2] = b >> 8


def unpack16(raw, kv_bits, scale, zero):
    """16 bytes of a token's row -> its dims in order, de-quantised: fma_T(T(q), scale, zero)."""
    if kv_bits == 16:
        return from_bits(raw[0::2].astype(np.uint16) | (raw[1::2].astype(np.uint16) << 8), F16)
    if kv_bits == 8:
        q = raw.astype(np.float32)
    else:
        q = []
        for w in raw.view(np.uint32):
            n = [(int(w) >> (4 * j)) & 15 for j in range(8)]
            q += [n[0], n[4], n[1], n[5], n[2], n[6], n[3], n[7]]       # cvt_u4x8 pairs nibbles (j, j + 4); the cache's order undoes it
        q = np.array(q, np.float32)
    return OA.t_fma(q, np.float32(scale), np.float32(zero), F16)


def load_tile(pool, kv_bits, block_len, Hkv, h, is_v, table, block_bytes, layer_offset, j, last):
    """One 128-key operand tile as the seven loader warps fill it."""
    row_bytes = D * kv_bits // 8
    units = row_bytes // 16
    tile = np.full(KEYS * D * 2, 0xA5, np.uint8)
    for w in range(LOADERS):
        for i in range(w, KEYS // 8 * (units // 4), LOADERS):
            for lane in range(32):
                row, unit = i // (units // 4) * 8 + (lane & 7), i % (units // 4) * 4 + (lane >> 3)
                key = j * KEYS + row
                raw, s, z = np.zeros(16, np.uint8), 0.0, 0.0
                if key <= last:
                    blk = table[key // block_len] * block_bytes + layer_offset
                    bt = key % block_len
                    at = blk + (2 * h + is_v) * block_len * row_bytes + bt * row_bytes + unit * 16
                    raw = pool[at:at + 16].copy()
                    if kv_bits != 16:
                        at = blk + Hkv * 2 * block_len * row_bytes + (2 * h + is_v) * block_len * 4 + bt * 4
                        s, z = from_bits(pool[at:at + 4].view(np.uint16), F16)
                x = unpack16(raw, kv_bits, s, z) if key <= last else np.zeros(16 * 8 // kv_bits, np.float32)
                for c in range(16 // kv_bits):
                    put16(tile, (unit * (16 // kv_bits) + c) * (KEYS * 16) + row * 16, x[8 * c:8 * c + 8])
    return tile


def emulate(pool, block_bytes, tables, cu_q, cu_k, layer_offset, block_len, Hq, Hkv, kv_bits, q_rot, qk_scale, ctas=0):
    G = Hq // Hkv
    TQ = ROWS // G
    T = cu_q[-1]
    out = np.zeros((T, Hq * D), np.float32)
    pieces = []                                                         # (sequence, first token, kv-head), places of the list before it
    place = 0
    for b in range(len(cu_q) - 1):
        q_len, hist = cu_q[b + 1] - cu_q[b], cu_k[b + 1] - cu_k[b] - (cu_q[b + 1] - cu_q[b])
        for q0 in range(0, q_len, 2 * TQ):
            n = (hist + min(q_len, q0 + 2 * TQ) - 1) // KEYS + 1
            for h in range(Hkv):
                pieces.append((b, q0, h, q_len, hist, n, place))
                place += START + n
    cuts = [place * c // ctas for c in range(1, ctas)]
    for b, q0, h, q_len, hist, n, first in pieces:
        # the piece's key tiles, cut where a range ends
        edges = sorted({0, n} | {min(n, max(0, c - first - START)) for c in cuts})
        last = hist + min(q_len, q0 + 2 * TQ) - 1
        kv = [[load_tile(pool, kv_bits, block_len, Hkv, h, v, tables[b], block_bytes, layer_offset, j, last) for v in (0, 1)] for j in range(n)]
        K = [read_operand(x[0], KEYS, D, KEYS * 16, 128).astype(np.float64) for x in kv]
        V = [read_mn_major(x[1], D, KEYS, 128, KEYS * 16).astype(np.float64) for x in kv]
        for t in range(2):
            nq = max(0, min(TQ, q_len - q0 - t * TQ))
            if nq == 0:
                continue
            r = np.arange(ROWS)
            tq, g = r // G, r % G
            valid = tq < nq
            pos0 = hist + q0 + t * TQ
            pos = np.where(valid, pos0 + tq, 0x7fffffff)
            tok = cu_q[b] + q0 + t * TQ + tq
            q_op = np.zeros(ROWS * D * 2, np.uint8)
            for row in np.nonzero(valid)[0]:
                for c in range(D // 8):
                    put16(q_op, (c * ROWS + row) * 16, q_rot[tok[row], h * G + g[row], c * 8:c * 8 + 8])
            Q = read_operand(q_op, ROWS, D, ROWS * 16, 128).astype(np.float64)
            tiles = (pos0 + nq - 1) // KEYS + 1                         # of this tile of rows
            M, L, O = np.full(ROWS, -np.inf), np.zeros(ROWS), np.zeros((ROWS, D))
            for j0, j1 in zip(edges, edges[1:]):
                m, l, o = np.full(ROWS, -np.inf), np.zeros(ROWS), np.zeros((ROWS, D))
                for j in range(j0, min(j1, tiles)):
                    S = (Q @ K[j].T).astype(np.float32)
                    S = np.where(j * KEYS + np.arange(KEYS)[None, :] <= pos[:, None], S, -np.inf)
                    m_new = np.maximum(m, S.max(1))
                    alpha = np.where(m == -np.inf, 0.0, np.exp2((m - np.where(m_new == -np.inf, 0.0, m_new)) * qk_scale))
                    mc = np.where(m_new == -np.inf, 0.0, m_new)
                    P = rn(np.exp2((S.astype(np.float64) - mc[:, None]) * qk_scale).astype(np.float32), F16).astype(np.float64)
                    l = l * alpha + P.sum(1)                            # of the rounded weights, as the product takes them
                    o = o * alpha[:, None] + P @ V[j]
                    m = m_new
                # parts in order; a part that holds no key of the row has no maximum
                with np.errstate(invalid="ignore"):
                    top = np.maximum(M, m)
                    a, w = np.where(M == -np.inf, 0.0, np.exp2((M - top) * qk_scale)), np.where(m == -np.inf, 0.0, np.exp2((m - top) * qk_scale))
                M, L, O = top, L * a + l * w, O * a[:, None] + o * w[:, None]
            res = rn((O[valid] / L[valid, None]).astype(np.float32), F16)
            for row, x in zip(np.nonzero(valid)[0], res):
                hq = h * G + g[row]
                out[tok[row], hq * D:(hq + 1) * D] = x
    return out


@pytest.mark.parametrize("kv_bits,heads,ctas", [(8, (4, 1), 0), (4, (4, 1), 0), (16, (4, 1), 0), (8, (2, 2), 0),
                                                (4, (6, 1), 0), (16, (6, 1), 0), (8, (4, 1), 16), (16, (2, 2), 16)])
def test_kernel_index_math_reproduces_the_oracle(kv_bits, heads, ctas):
    Hq, Hkv = heads
    rng = np.random.default_rng(kv_bits * 10 + Hq)
    q_lens, hists = np.array([37, 1, 70]), np.array([0, 70, 30])
    k_lens = q_lens + hists
    block_len, layers, layer = 64, 2, 1
    layout = OA.KvLayout(Hkv, block_len, D, kv_bits)
    blocks_per = [(int(k) + block_len - 1) // block_len for k in k_lens]
    nblk = sum(blocks_per) + 1
    cache = OA.PagedKvCache(nblk, layers, layout, F16)
    cache.pool[:] = rng.integers(0, 256, cache.pool.shape, dtype=np.uint8)       # garbage, incl. NaN bit patterns
    perm = rng.permutation(nblk)
    tables, o = [], 0
    for n in blocks_per:
        tables.append(perm[o:o + n].tolist())
        o += n
    rope = OA.RopeParam(type=OA.ROPE_DEFAULT, dim=D, base=1e4)
    for b, hlen in enumerate(hists):
        if hlen:
            OA.process_kv(cache, tables[b], layer, 0, rn(rng.standard_normal((hlen, Hkv, D)).astype(np.float32), F16),
                          rn(rng.standard_normal((hlen, Hkv, D)).astype(np.float32), F16), rope)
    T = int(q_lens.sum())
    qkv = rn(rng.standard_normal((T, (Hq + 2 * Hkv) * D)).astype(np.float32), F16)
    ref = OA.prefill_attention(qkv, cache, tables, q_lens, k_lens, layer, Hq, Hkv, rope)      # also writes the chunk's K/V
    # what the prologue kernel hands the attention kernel: rotated Q (the pages were just written by the oracle)
    q_rot = np.zeros((T, Hq, D), np.float32)
    t0 = 0
    for b, ql in enumerate(q_lens):
        pos = (hists[b] + np.arange(ql))[:, None]
        q_rot[t0:t0 + ql] = OA.apply_rope(qkv[t0:t0 + ql, :Hq * D].reshape(ql, Hq, D), np.broadcast_to(pos, (ql, Hq)), rope, F16)
        t0 += ql
    cu_q = np.concatenate([[0], np.cumsum(q_lens)]).tolist()
    cu_k = np.concatenate([[0], np.cumsum(k_lens)]).tolist()
    c = float(np.float32(np.float32(1.4426950408889634) / np.float32(np.sqrt(np.float32(D)))))
    got = emulate(cache.pool.reshape(-1), cache.block_bytes, tables, cu_q, cu_k, cache.layer_offset(layer), block_len, Hq, Hkv,
                  kv_bits, q_rot, c, ctas)
    assert np.isfinite(got).all()
    # tiled online softmax vs the oracle's single pass: a few fp16 ulps of an O(1) output
    assert np.abs(got - ref).max() <= 2e-3
