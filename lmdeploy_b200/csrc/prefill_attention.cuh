// Paged-KV causal prefill ("context") attention for sm_100a.
//
// Stands where the reference runs, for a chunk of q_len > 1 new tokens per sequence,
//   invokeProcessKV_v2  (kv_cache_utils_v2.cu:18-210)   -> prefill_prologue_kernel (decode_attention.cu)
//   invokeFlattenKV_v2  (kv_cache_utils_v2.cu:212-420)  -> fused here: pages are de-quantised into the operand tiles
//   dispatchAttention   (attention.cu, attention_universal.h:355-553 with the sm80 prefill mainloop)
// Not a port: S = Q.K^T and O += P.V run on tcgen05 tensor cores with fp32 accumulators in tensor memory.
//
// A UNIT is one sequence's block of up to 2 x (128 / G) query tokens; with one kv-head it makes two UMMA tiles of 128 rows
// (row = token_in_tile * G + head_in_group), so every K/V tile fetched and de-quantised from the pages serves both tiles and all
// heads of the group.  Roles of a CTA (one per SM, persistent):
//   warps 0-3 / 4-7   softmax of tile 0 / 1, thread = row: scores from TMEM, causal mask, base-2 online softmax, P (T) back to
//                     TMEM as the A operand of P.V, in two halves so that the first half's P.V runs under the second half's
//                     exponentials; the accumulator stays in TMEM and is rescaled when the maximum of a row of the warp has grown.
//                     A warp's exponentials and those of its neighbour in the other tile take turns
//   warp 8            issues every tcgen05.mma: Q.K^T of tile t for the next keys right behind P.V of tile t, so that the tensor
//                     pipe works on one tile while the other one is in its softmax
//   warps 9-15        K/V pages -> operand tiles of 128 keys (two-slot rings), and a piece's queries: T rows by asynchronous copies;
//                     int8/int4 by asynchronous copies into a staging tile (every thread reads back its own bytes only), then with
//                     the decode kernel's arithmetic (exact int -> T, one T fma with the token's (scale, zero)) into the ring.
//                     All operand tiles have rows of 128 bytes in the tensor core's 128-byte swizzle (prefill_offset): K-major for Q.K^T, V MN-major
// Work: all (unit, kv-head, 128-key tile) triples form one flat list that is cut into equal ranges, one per CTA; a (unit, kv-head)
// whose keys fall into several ranges leaves fp32 partials (accumulator, row maximum, row sum) that prefill_merge_kernel combines in
// CTA order (deterministic).  So a chunk of a few tokens over a long history uses every SM, and unequal prompts end together.
// Precision: weights relative to the true maximum so far, not to one that may lag (the largest weight of a row is then one, which
// rounding to T leaves alone), and summed as T rounds them (numerator and denominator alike).  Error against 64 bits, prompts of 2048,
// 1190 and 2048 tokens, f16 / bf16 pages: 3.42e-4 / 2.66e-3; with a maximum that may lag by 2^8 and the sum of the unrounded weights
// 3.47e-4 / 2.70e-3; one CTA per 128 rows with a maximum per 64 keys had 3.43e-4 / 2.67e-3.
// Measured (B200, whole operator, short runs; prompts of 2048, 1190 and 2048 tokens, f16 pages, 32 / 8 heads / one prompt of 2048 behind 4096):
//   one CTA per 128 rows, 64-key tiles, the phases one after another                                                465 us
//   this design with operand tiles [d/8][row][8], which scatter a row's line over 16 lines of shared memory:
//   16-byte copies then enter it at one per cycle and SM, 4 k cycles for the 64 KB of a 256 x 128 step              168 / 221 us
//   the same, queries fetched by the loaders a piece ahead (3 us of each piece before), outputs read at once        166 / 224
//   128-byte swizzle: eight lanes copy a line to a line                                                             144 / 189  (148 / 197 without the turns)
//   two floats per multiplication, fewer instructions per copy, columns of a rescale read ahead                     140 / 186
//   the prologue's heads by kind, a merge with 16 dims a thread                                                    131 / 182
// All of them agree bit for bit.  A step takes some 4 k cycles where the tensor pipe needs 2.0 k and the exponentials 2.0 k: the chain of
// a tile (scores, maximum, rescaled accumulator, weights: 64 % of all issue slots) bounds it.  Without any rescale 170 us, without any exponential
// 171 (one prompt of 2048 behind 4096, 189 with both).
#pragma once

#include "common.cuh"
#include "prefill_work.cuh"
#include "umma.cuh"

namespace b200 {
namespace attn {

constexpr int kPfThreads  = 32 * (8 + 1 + kPfLoaders);  // 16 warps: 128 registers a thread at launch
constexpr int kPfTile     = kPfKeys * kPfD * 2;  // bytes of a Q, K or V operand tile
constexpr int kPfStages   = 2;
constexpr int kPfColS = 0, kPfColO = 256, kPfTmemCols = 512;  // tile t: S / P at t * 128, O at 256 + t * 128

// dynamic shared memory: Q tiles, K and V rings, and the staging tiles of quantised pages
template<int KVBITS>
constexpr int kPfSmem = (2 + 2 * kPfStages) * kPfTile + (KVBITS == 16 ? 0 : 2 * kPfKeys * kPfD * KVBITS / 8);

// partial of one (CTA range end, tile): accumulator [d/4][row] float4, then (max, sum) [row] float2
constexpr size_t kPfPartialFloats = (size_t)kPfRows * kPfD + 2 * kPfRows;

// Units and their places, by one block of THREADS threads; thread = sequence.
template<int THREADS>
B200_DEVICE void prefill_plan(const PrefillParams& p)
{
    __shared__ int2 s_warp[THREADS / 32];
    __shared__ int2 s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int TQ2 = prefill_unit_tokens(p);
    if (tid == 0) {
        s_base = make_int2(0, 0);
    }
    __syncthreads();
    for (int b0 = 0; b0 < p.batch; b0 += THREADS) {
        const int b = b0 + tid;
        int       q_len = 0, hist = 0, tok0 = 0;
        if (b < p.batch) {
            tok0  = p.cu_q_len[b];
            q_len = p.cu_q_len[b + 1] - tok0;
            hist  = p.cu_k_len[b + 1] - p.cu_k_len[b] - q_len;
        }
        int2 v = make_int2(0, 0);  // (units, places)
        for (int q0 = 0; q0 < q_len; q0 += TQ2) {
            v.x += 1;
            v.y += prefill_places(hist, q_len, q0, TQ2);
        }
        int2 s = v;  // inclusive scan
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, s.x, o), y = __shfl_up_sync(0xffffffffu, s.y, o);
            if (lane >= o) {
                s.x += x, s.y += y;
            }
        }
        if (lane == 31) {
            s_warp[warp] = s;
        }
        __syncthreads();
        int2 base = s_base;
        for (int w = 0; w < warp; ++w) base.x += s_warp[w].x, base.y += s_warp[w].y;
        int u = base.x + s.x - v.x, t = base.y + s.y - v.y;
        for (int q0 = 0; q0 < q_len; q0 += TQ2) {
            const int n  = prefill_places(hist, q_len, q0, TQ2);
            p.units[u++] = PrefillUnit{t, n, b, q0, tok0, q_len, hist, 0};
            t += n;
        }
        __syncthreads();
        if (tid == THREADS - 1) {
            s_base = make_int2(base.x + s.x, base.y + s.y);
        }
        __syncthreads();
    }
    if (tid == 0) {
        p.units[s_base.x] = PrefillUnit{s_base.y, 0, p.batch, 0, 0, 0, 0, 0};
    }
    __syncthreads();
    for (int c = tid; c < p.main_ctas; c += THREADS) {
        p.ranges[c] = prefill_range(p, s_base.x, s_base.y, c);
    }
}

B200_DEVICE void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// One key tile as the loaders see it: where its two 64-key halves lie (block_len is a multiple of 64: a half lies in one page); V
// follows K by *_step bytes.  Keys past `last` (the newest that any query of the unit sees) may be uninitialised: they become zeros.
struct PrefillKeyTile {
    int         h, j, j1, last;
    char**      blocks;  // the sequence's block table
    const char *data0, *data1, *param0, *param1;

    B200_DEVICE void begin(const PrefillParams& p, const PrefillSegment& s, int TQ)
    {
        blocks = p.block_ptrs + p.cu_block_nums[s.b];
        h = s.h, j = s.j0, j1 = s.j1;
        last = s.hist + min(s.q_len, s.q0 + 2 * TQ) - 1;
    }
    // the first half is always there (its first key is visible to some query); past `last` the block table may have ended
    B200_DEVICE void find(const PrefillParams& p, int row_bytes)
    {
        at(p, j * kPfKeys, row_bytes, data0, param0);
        data1 = data0, param1 = param0;
        if (j * kPfKeys + 64 <= last) {
            at(p, j * kPfKeys + 64, row_bytes, data1, param1);
        }
    }
    B200_DEVICE void at(const PrefillParams& p, int key, int row_bytes, const char*& data, const char*& param) const
    {
        const int   i   = key / p.block_len, bt = key - i * p.block_len;
        const char* blk = blocks[i] + p.layer_offset;
        data            = blk + (size_t)(h * 2) * p.block_len * row_bytes + (size_t)bt * row_bytes;
        param           = blk + ((size_t)p.num_kv_heads * 2 * row_bytes + h * 2 * 4) * p.block_len + bt * 4;
    }
};

// Loader warps: rows of K or of V (PrefillRowMap says which)
template<class T, int KVBITS>
struct PrefillRows: PrefillRowMap<KVBITS> {
    using Map = PrefillRowMap<KVBITS>;
    using Map::half_of;
    using Map::key_of;
    using Map::unit_of;
    static constexpr int kRow = Map::kRow, kInstr = Map::kInstr, kIter = Map::kIter;
    uint32_t par[kIter];  // (scale, zero) of the thread's rows

    // asynchronous 16-byte copies of the tile's rows into the staging tile `dst`, where instruction i of the tile has 512 bytes of its own
    B200_DEVICE void fetch(const PrefillParams& p, const PrefillKeyTile& x, int is_v, uint32_t dst, int w, int lane)
    {
#pragma unroll
        for (int it = 0; it < kIter; ++it) {
            if (w + kPfLoaders * it >= kInstr) {
                break;
            }
            const int      row  = key_of(w, lane, it), unit = unit_of(w, lane, it);
            const bool     live = x.j * kPfKeys + row <= x.last, half = half_of(w, it);
            const char*    src  = (half ? x.data1 : x.data0) + is_v * p.block_len * kRow + (live ? (row & 63) * kRow : 0) + unit * 16;
            cp_async16(dst + (w + kPfLoaders * it) * 512 + lane * 16, src, live ? 16 : 0);
            par[it] = live ? *reinterpret_cast<const uint32_t*>((half ? x.param1 : x.param0) + is_v * p.block_len * 4 + (row & 63) * 4) : 0u;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // staging tile -> T rows of the operand tile
    B200_DEVICE void convert(uint32_t staging, uint32_t tile, int w, int lane) const
    {
        using Ops = TypeOps<T>;
#pragma unroll
        for (int it = 0; it < kIter; ++it) {
            if (w + kPfLoaders * it >= kInstr) {
                break;
            }
            const uint4    raw = lds128(staging + (w + kPfLoaders * it) * 512 + lane * 16);
            const int      key = key_of(w, lane, it);
            const int      c0  = unit_of(w, lane, it) * (16 / KVBITS);  // first 8-dim chunk of the unit
            const uint32_t s2 = __byte_perm(par[it], par[it], 0x1010), z2 = __byte_perm(par[it], par[it], 0x3232);
#pragma unroll
            for (int k = 0; k < 16 / KVBITS; ++k) {
                uint32_t r[4];
                if constexpr (KVBITS == 8) {
                    Ops::cvt_u8x4(k ? raw.z : raw.x, r[0], r[1]);
                    Ops::cvt_u8x4(k ? raw.w : raw.y, r[2], r[3]);
                }
                else {
                    // one u32 = 8 dims, nibble j holds element [0,2,4,6,1,3,5,7][j]; cvt_u4x8 pairs nibbles (j, j+4) = dims (2j, 2j+1)
                    Ops::cvt_u4x8((&raw.x)[k], r);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) r[i] = Ops::fma2(r[i], s2, z2);
                sts128(tile + prefill_offset(c0 + k, key), r[0], r[1], r[2], r[3]);
            }
        }
    }
};

// ... T rows (PrefillLineMap), straight into the operand tile `dst`
template<class T>
struct PrefillRows<T, 16> {
    using Map = PrefillLineMap;
    static constexpr int kRow = kPfD * 2;

    B200_DEVICE void fetch(const PrefillParams& p, const PrefillKeyTile& x, int is_v, uint32_t dst, int w, int lane)
    {
        const uint32_t to   = dst + Map::place(w, lane);
        const int64_t  from = is_v * p.block_len * kRow + Map::unit0(lane) * 16;
        const int      last = x.last - x.j * kPfKeys;
#pragma unroll
        for (int it = 0; it < Map::kIter; ++it) {
            const int row = Map::row_of(w, lane, it);
            if (it + 1 == Map::kIter && !Map::inside(w, it)) {
                break;
            }
            const int      n   = row <= last ? 16 : 0;
            const char*    src = (Map::row_of(w, 0, it) < 64 ? x.data0 : x.data1) + from + (n ? (row & 63) * kRow : 0);
            const uint32_t at  = Map::step(to, it);
            cp_async16(at, src, n);
            cp_async16(at + kPfTile / 2, src + 128, n);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
};

// Loader warps: the query rows of a piece
struct PrefillQueries {
    int tok, n0, n1, h;  // first token; tokens of the two tiles; kv-head

    B200_DEVICE void begin(const PrefillSegment& s, int TQ) { tok = s.tok0 + s.q0, n0 = s.tokens(0, TQ), n1 = s.tokens(1, TQ), h = s.h; }
    // asynchronous copies, one group; rows without a token become zeros
    template<class T>
    B200_DEVICE void fetch(const PrefillParams& p, int G, int TQ, uint32_t dst, int w, int lane) const
    {
        using Map = PrefillLineMap;
        static_assert(kPfRows == kPfKeys);
#pragma unroll 1
        for (int t = 0; t < 2; ++t) {
            const int n = t ? n1 : n0;
            if (n == 0) {
                break;
            }
            const uint32_t to = dst + t * kPfTile + Map::place(w, lane);
#pragma unroll 1
            for (int it = 0; it < Map::kIter && Map::inside(w, it); ++it) {
                const int      row = Map::row_of(w, lane, it), tr = row / G, live = tr < n ? 16 : 0;
                const T*       src = reinterpret_cast<const T*>(p.q_rot) + ((size_t)(tok + t * TQ + (live ? tr : 0)) * p.num_heads + (size_t)h * G + (row - tr * G)) * kPfD + Map::unit0(lane) * 8;
                const uint32_t at  = Map::step(to, it);
                cp_async16(at, src, live);
                cp_async16(at + kPfTile / 2, src + kPfD / 2, live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
};

// two floats at once, each rounded by itself
B200_DEVICE uint64_t pair2(float2 x)
{
    uint64_t y;
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(x.x), "f"(x.y));
    return y;
}
B200_DEVICE float2 pair2(uint64_t x)
{
    float2 y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(y.x), "=f"(y.y) : "l"(x));
    return y;
}
B200_DEVICE float2 fma2(float2 a, float2 b, float2 c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pair2(a)), "l"(pair2(b)), "l"(pair2(c)));
    return pair2(d);
}
B200_DEVICE float2 mul2(float2 a, float2 b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pair2(a)), "l"(pair2(b)));
    return pair2(d);
}
B200_DEVICE float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// SPLIT: p.partial is there; else whole pieces (a kernel of its own: both walks in one cost registers, 181 -> 194 us on the
// prompts above).  The split form is at its 128 registers and spills 40 bytes, the whole one does not spill.
template<class T, int KVBITS, bool SPLIT>
__global__ void __launch_bounds__(kPfThreads, 1) prefill_attention_kernel(const PrefillParams p)
{
    using Ops = TypeOps<T>;
    extern __shared__ __align__(1024) uint8_t pf_smem[];
    __shared__ uint64_t bar_q, bar_qfree;                            // a piece's Q tiles are there, its last Q.K^T has read them
    __shared__ uint64_t bar_s[2], bar_p[4], bar_o[2];                // per tile: scores ready, halves of P ready, P.V done
    __shared__ uint64_t bar_full[2 * kPfStages], bar_empty[2 * kPfStages];                     // rings of K, then of V
    __shared__ uint32_t s_tmem;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = tid & 31;
    const int G  = p.num_heads / p.num_kv_heads;
    const int TQ = kPfRows / G;  // query tokens per tile

    pdl_launch_dependents();
    if (warp == 8) {
        umma::tmem_alloc(smem_u32(&s_tmem), kPfTmemCols);
    }
    if (tid < 2) {
        mbar_init(smem_u32(tid ? &bar_qfree : &bar_q), tid ? 1 : kPfLoaders);
        mbar_init(smem_u32(&bar_s[tid]), 1);
        mbar_init(smem_u32(&bar_p[tid]), 4);  // one arrival per warp
        mbar_init(smem_u32(&bar_p[2 + tid]), 4);
        mbar_init(smem_u32(&bar_o[tid]), 1);
#pragma unroll
        for (int i = tid; i < 2 * kPfStages; i += 2) {
            mbar_init(smem_u32(&bar_full[i]), kPfLoaders);
            mbar_init(smem_u32(&bar_empty[i]), 1);
        }
        fence_mbar_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    pdl_wait();  // q_rot, the chunk's K/V pages and the units come from the prologue kernel
    const uint32_t tmem = s_tmem;
    const uint32_t q_op = smem_u32(pf_smem), k_op = q_op + 2 * kPfTile, v_op = k_op + kPfStages * kPfTile;

    PrefillWalk<SPLIT> walk(p, blockIdx.x);
    PrefillSegment     s{};

    if (warp > 8) {
        // ================================ loaders ================================
        umma::set_max_registers_dec<64>();
        using Rows           = PrefillRows<T, KVBITS>;
        const int      w     = warp - 9;
        uint32_t       count = 0;  // tiles so far: slot = count % 2, lap = count / 2
        const uint32_t full0 = smem_u32(&bar_full[0]), empty0 = smem_u32(&bar_empty[0]);  // [is_v][slot]
        auto           publish = [&](uint32_t bar) {
            fence_proxy_async();  // generic-proxy stores -> visible to the tensor core's async-proxy reads
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar);
            }
        };
        PrefillKeyTile x, y;  // this tile; the next one, looked up a tile ahead of its use
        auto           step = [&](const PrefillKeyTile& from, PrefillKeyTile& to) {
            to.j = from.j + 1, to.j1 = from.j1, to.blocks = from.blocks, to.h = from.h, to.last = from.last;
            if (to.j >= to.j1) {
                if (!walk.next(s)) {
                    return false;
                }
                to.begin(p, s, TQ);
            }
            to.find(p, Rows::kRow);
            return true;
        };
        // A piece's Q tiles, fetched behind its first keys: the earlier piece's last softmax is under way then
        PrefillQueries queries;
        bool           first = true;
        uint32_t       phq   = 1;
        auto           fetch_q = [&] {
            mbar_wait(smem_u32(&bar_qfree), phq);
            phq ^= 1;
            queries.fetch<T>(p, G, TQ, q_op, w, lane);
        };
        bool more = walk.next(s);
        if (more) {
            x.begin(p, s, TQ);
            x.find(p, Rows::kRow);
            queries.begin(s, TQ);
        }
        if constexpr (KVBITS == 16) {
            // copy groups K0 V0 K1 V1 ..: a group is published when the next one has been issued (three in flight measured slower: the
            // copies then hold up the other warps' shared-memory traffic)
            Rows     rows;
            uint32_t waiting = 0;
            while (more) {
                const uint32_t slot = count % kPfStages, ph = (count / kPfStages) & 1;
                const bool     ends = x.j + 1 >= x.j1;
                more                = step(x, y);
#pragma unroll
                for (int is_v = 0; is_v < 2; ++is_v) {
                    const uint32_t ring = (is_v * kPfStages + slot) * 8;
                    mbar_wait(empty0 + ring, ph ^ 1);
                    rows.fetch(p, x, is_v, (is_v ? v_op : k_op) + slot * kPfTile, w, lane);
                    if (waiting) {
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                        publish(waiting);
                    }
                    waiting = full0 + ring;
                    if (!is_v && first) {
                        fetch_q();
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                        publish(waiting);
                        waiting = smem_u32(&bar_q);
                    }
                }
                x     = y;
                first = ends;
                if (ends && more) {
                    queries.begin(s, TQ);
                }
                ++count;
                if (ends) {  // the last tile of a piece must not wait for the next piece, whose keys may have to wait for its P.V
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    publish(waiting);
                    waiting = 0;
                }
            }
        }
        else {
            const uint32_t stage = v_op + kPfStages * kPfTile;
            Rows           rows[2];
            if (more) {
                rows[0].fetch(p, x, 0, stage, w, lane);
                rows[1].fetch(p, x, 1, stage + kPfKeys * Rows::kRow, w, lane);
            }
            while (more) {
                const uint32_t slot = count % kPfStages, ph = (count / kPfStages) & 1;
                const bool     ends = x.j + 1 >= x.j1;
                more = step(x, y);
                if (first) {
                    fetch_q();
                }
#pragma unroll
                for (int is_v = 0; is_v < 2; ++is_v) {
                    const uint32_t ring = (is_v * kPfStages + slot) * 8, from = stage + is_v * kPfKeys * Rows::kRow;
                    if (!is_v && first) {
                        asm volatile("cp.async.wait_group 2;" ::: "memory");  // behind K: V and the queries
                    }
                    else {
                        asm volatile("cp.async.wait_group 1;" ::: "memory");  // this tile's bytes are there (the other matrix's may not be)
                        if (first) {
                            publish(smem_u32(&bar_q));
                        }
                    }
                    mbar_wait(empty0 + ring, ph ^ 1);
                    rows[is_v].convert(from, (is_v ? v_op : k_op) + slot * kPfTile, w, lane);
                    publish(full0 + ring);
                    if (more) {
                        rows[is_v].fetch(p, y, is_v, from, w, lane);  // the thread has read its bytes (their conversions are stored)
                    }
                    else {
                        asm volatile("cp.async.commit_group;" ::: "memory");  // keeps the count of groups behind wait_group
                    }
                }
                x     = y;
                first = ends;
                if (ends && more) {
                    queries.begin(s, TQ);
                }
                ++count;
            }
        }
    }
    else if (warp == 8) {
        // ================================ MMA issue ================================
        umma::set_max_registers_dec<64>();
        constexpr bool     kBf   = std::is_same<T, nv_bfloat16>::value;
        constexpr uint32_t kQk   = umma::make_idesc_f16(kPfRows, kPfKeys, kBf);
        constexpr uint32_t kPv   = umma::make_idesc_f16(kPfRows, kPfD, kBf) | (1u << 16);  // B is MN-major
        uint32_t count = 0, phq = 0, php[2] = {0, 0};
        auto qk = [&](int t, uint32_t slot) {
            const uint64_t ad = umma::make_smem_desc_sw128(q_op + t * kPfTile, 16, 1024);
            const uint64_t bd = umma::make_smem_desc_sw128(k_op + slot * kPfTile, 16, 1024);
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < kPfD / 16; ++ks) {
                    const uint64_t at = (uint64_t)(prefill_offset(2 * ks, 0) >> 4);  // 16 dims: two chunks
                    umma::mma_f16_ss(tmem + kPfColS + t * 128, ad + at, bd + at, kQk, ks > 0);
                }
                umma::commit(smem_u32(&bar_s[t]));
            }
            __syncwarp();
        };
        while (walk.next(s)) {
            const int n = s.j1 - s.j0, cnt[2] = {s.tiles(0, TQ), s.tiles(1, TQ)};
            mbar_wait(smem_u32(&bar_full[count % kPfStages]), (count / kPfStages) & 1);
            mbar_wait(smem_u32(&bar_q), phq);
            phq ^= 1;
            umma::fence_after_sync();
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (cnt[t] > 0) {
                    qk(t, count % kPfStages);
                }
            }
            if (elect_one()) {
                umma::commit(smem_u32(&bar_empty[count % kPfStages]));
                if (n == 1) {
                    umma::commit(smem_u32(&bar_qfree));
                }
            }
            __syncwarp();
            for (int i = 0; i < n; ++i, ++count) {
                const uint32_t slot = count % kPfStages, ph = (count / kPfStages) & 1;
                const uint32_t next = (count + 1) % kPfStages, phn = ((count + 1) / kPfStages) & 1;
                mbar_wait(smem_u32(&bar_full[kPfStages + slot]), ph);
                umma::fence_after_sync();
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (i < cnt[t]) {
                        // V tile as MN-major operand: 64-dim groups half a tile apart (LBO), 8-key groups 1024 bytes apart (SBO)
                        const uint64_t bd = umma::make_smem_desc_sw128(v_op + slot * kPfTile, kPfTile / 2, 1024);
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            mbar_wait(smem_u32(&bar_p[2 * half + t]), php[t]);
                            umma::fence_after_sync();
                            if (elect_one()) {
#pragma unroll
                                for (int ks = 4 * half; ks < 4 * half + 4; ++ks) {
                                    umma::mma_f16_ts(tmem + kPfColO + t * 128, tmem + kPfColS + t * 128 + ks * 8, bd + (uint64_t)(ks * (16 * 128 >> 4)), kPv,
                                                     i > 0 || ks > 0);
                                }
                                if (half) {
                                    umma::commit(smem_u32(&bar_o[t]));
                                }
                            }
                            __syncwarp();
                        }
                        php[t] ^= 1;
                    }
                    if (t == 1 && elect_one()) {
                        umma::commit(smem_u32(&bar_empty[kPfStages + slot]));
                    }
                    __syncwarp();
                    if (i + 1 < n) {
                        if (t == 0) {
                            mbar_wait(smem_u32(&bar_full[next]), phn);
                            umma::fence_after_sync();
                        }
                        if (i + 1 < cnt[t]) {
                            qk(t, next);  // its scores replace the P that the P.V just issued reads: the pipe runs them in order
                        }
                        if (t == 1 && elect_one()) {
                            umma::commit(smem_u32(&bar_empty[next]));
                            if (i + 2 == n) {
                                umma::commit(smem_u32(&bar_qfree));
                            }
                        }
                        __syncwarp();
                    }
                }
            }
        }
    }
    else {
        // ================================ softmax: thread = row of tile t ================================
        umma::set_max_registers_inc<192>();  // 256 x 192 + 256 x 64 = the 512 x 128 of the launch
        const int      t  = warp >> 2, r = tid & 127;
        const int      tq = r / G, g = r - tq * G;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t ts = lanes + kPfColS + t * 128, to = lanes + kPfColO + t * 128;
        const float    c = p.qk_scale;
        uint32_t       phs = 0, pho = 0;  // parity of the next score / accumulator phase
        auto           arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(bar));
            }
        };
        // The exponentials of a warp and of its neighbour in the other tile, on the same scheduler, take turns (barriers 1 - 4 / 5 - 8: tile 0's /
        // tile 1's turn): side by side both would end late, and the tensor pipe would have nothing to do meanwhile.  `both` steps of a piece have both.
        const int turn = 1 + (warp & 3);
        if (t == 1) {
            named_bar_arrive(turn, 64);
        }
        while (walk.next(s)) {
            const int    nq = s.tokens(t, TQ), cnt = s.tiles(t, TQ), both = min(s.tiles(0, TQ), s.tiles(1, TQ));
            const bool   valid = tq < nq;  // rows >= TQ * G (G not a power of two) have tq >= TQ >= nq
            const int    pos0  = s.hist + s.q0 + t * TQ;
            const int    pos_q = valid ? pos0 + tq : 0x7fffffff;  // padding rows see everything (finite softmax, never stored)
            const size_t tok   = (size_t)s.tok0 + s.q0 + t * TQ + tq;
            const int    h = s.h, j0 = s.j0;
            const bool   whole = !SPLIT || (s.j0 == 0 && s.j1 == s.n);
            float        m = -INFINITY, l = 0.f;
            for (int i = 0; i < cnt; ++i) {
                const int  key0 = (j0 + i) * kPfKeys;
                const bool mask = key0 + kPfKeys - 1 > pos0;  // some row of the tile does not see some key
                mbar_wait(smem_u32(&bar_s[t]), phs);
                phs ^= 1;
                umma::fence_after_sync();
                // the row's 128 scores in registers: TMEM is read once
                uint32_t v[kPfKeys / 32][32];
#pragma unroll
                for (int ch = 0; ch < kPfKeys / 32; ++ch) umma::ld_32x32b_x32(ts + ch * 32, v[ch]);
                umma::wait_ld();
                if (mask) {
#pragma unroll
                    for (int k = 0; k < kPfKeys; ++k) {
                        if (key0 + k > pos_q) {
                            v[k >> 5][k & 31] = __float_as_uint(-INFINITY);
                        }
                    }
                }
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int k = 0; k < kPfKeys; k += 2) mx4[(k >> 1) & 3] = max3(mx4[(k >> 1) & 3], __uint_as_float(v[k >> 5][k & 31]), __uint_as_float(v[k >> 5][(k & 31) + 1]));
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                if (i == 0) {
                    m = mx;
                }
                else {
                    const float m_new = fmaxf(m, mx);
                    if (__any_sync(0xffffffffu, m_new > m)) {
                        const float alpha = m == -INFINITY ? 0.f : exp2_approx((m - m_new) * c);
                        mbar_wait(smem_u32(&bar_o[t]), pho ^ 1);  // P.V of the previous tile has completed
                        umma::fence_after_sync();
                        // the next columns are read while these are multiplied and written
                        uint32_t     o[2][16];
                        const float2 alpha2 = make_float2(alpha, alpha);
                        umma::ld_32x32b_x16(to, o[0]);
#pragma unroll
                        for (int ch = 0; ch < kPfD / 16; ++ch) {
                            uint32_t(&x)[16] = o[ch & 1];
                            umma::wait_ld();
                            if (ch + 1 < kPfD / 16) {
                                umma::ld_32x32b_x16(to + (ch + 1) * 16, o[(ch + 1) & 1]);
                            }
#pragma unroll
                            for (int k = 0; k < 16; k += 2) {
                                const float2 y = mul2(make_float2(__uint_as_float(x[k]), __uint_as_float(x[k + 1])), alpha2);
                                x[k] = __float_as_uint(y.x), x[k + 1] = __float_as_uint(y.y);
                            }
                            umma::st_32x32b_x16(to + ch * 16, x);
                        }
                        l *= alpha;
                        m = m_new;
                    }
                }
                if (i < both) {
                    named_bar_sync(turn + 4 * t, 64);
                }
                const float mc    = m == -INFINITY ? 0.f : m * c;
                const float2 c2 = make_float2(c, c), mc2 = make_float2(-mc, -mc);
                float        l4[4] = {0.f, 0.f, 0.f, 0.f};  // sums of the weights as T rounds them
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t pk[32];
#pragma unroll
                    for (int k = 0; k < 64; k += 2) {
                        const uint32_t(&x)[32] = v[2 * half + (k >> 5)];
                        const float2 e = fma2(make_float2(__uint_as_float(x[k & 31]), __uint_as_float(x[(k & 31) + 1])), c2, mc2);
                        pk[k >> 1] = Ops::pack2(exp2_approx(e.x), exp2_approx(e.y));  // column c of P holds keys (2c, 2c + 1)
                        Ops::add_pair(l4[(k >> 1) & 3], pk[k >> 1]);
                    }
                    umma::st_32x32b_x32(ts + half * 32, pk);
                    umma::wait_st();
                    umma::fence_before_sync();
                    arrive(&bar_p[2 * half + t]);
                }
                if (i < both) {
                    named_bar_arrive(turn + 4 * (1 - t), 64);
                }
                l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
                pho ^= 1;
            }
            if (cnt > 0) {
                mbar_wait(smem_u32(&bar_o[t]), pho ^ 1);
                umma::fence_after_sync();
            }
            if (whole) {
                // ---- whole piece: out = O / L ----
                if (cnt > 0) {
                    const float inv = 1.f / l;
                    T*          dst = reinterpret_cast<T*>(p.out) + tok * p.out_stride + ((size_t)h * G + g) * kPfD;
                    const bool  wide = (((uintptr_t)p.out | (uintptr_t)(p.out_stride * sizeof(T))) & 31) == 0;
                    uint32_t    v[kPfD / 32][32];
#pragma unroll
                    for (int ch = 0; ch < kPfD / 32; ++ch) umma::ld_32x32b_x32(to + ch * 32, v[ch]);
                    umma::wait_ld();
                    if (valid) {
#pragma unroll
                        for (int ch = 0; ch < kPfD / 16; ++ch) {
                            uint32_t x[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const int at = (ch & 1) * 16 + 2 * k;
                                x[k] = Ops::pack2(__uint_as_float(v[ch >> 1][at]) * inv, __uint_as_float(v[ch >> 1][at + 1]) * inv);
                            }
                            store_words8(dst + ch * 16, x, wide);
                        }
                    }
                }
            }
            else if (nq > 0) {
                // ---- part of a piece ----
                float* dst = p.partial + ((size_t)prefill_slot(blockIdx.x, j0) * 2 + t) * kPfPartialFloats;
                if (cnt > 0) {
                    uint32_t v[kPfD / 32][32];
#pragma unroll
                    for (int ch = 0; ch < kPfD / 32; ++ch) umma::ld_32x32b_x32(to + ch * 32, v[ch]);
                    umma::wait_ld();
#pragma unroll
                    for (int k = 0; k < kPfD / 4; ++k) {
                        const uint32_t* x = &v[k >> 3][4 * (k & 7)];
                        __stcg(reinterpret_cast<uint4*>(dst) + k * kPfRows + r, make_uint4(x[0], x[1], x[2], x[3]));
                    }
                }
                __stcg(reinterpret_cast<float2*>(dst + (size_t)kPfRows * kPfD) + r, make_float2(m, l));
            }
        }
        if (t == 0) {
            named_bar_sync(turn, 64);  // the turn that tile 1 gave back last
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 8) {
        umma::tmem_dealloc(tmem, kPfTmemCols);
    }
}

// Combines the partials of every (unit, kv-head) whose keys fell into several CTAs.  grid (CTA, 2 tiles, 4 x 32 dims): the block of
// the first CTA whose range begins inside the piece does the work; thread = row and 16 of the 32 dims, parts in CTA order.
// 16 dims a thread: with 8 dims and twice the blocks, each of which looks its piece up and reads the maxima and sums of all parts again, prompts take 2 us more,
// 4 x 400 - 512 tokens behind 300 - 1000 keys 95.8 instead of 94.0, 8 x 16 behind 3000 - 4000 56.4 instead of 54.6 (32 dims: 141, 95.3 and 54.3).  Registers
// go from 72 to 109, resident blocks from three to two per SM: four fillings of the SMs for 148 ranges, where it was five.
constexpr int kPfMergeThreads = 256, kPfMergeZ = 4;

template<class T>
__global__ void __launch_bounds__(kPfMergeThreads) prefill_merge_kernel(const PrefillParams p)
{
    using Ops = TypeOps<T>;
    pdl_launch_dependents();
    pdl_wait();
    const int    t = blockIdx.y;
    PrefillParts x;
    if (!prefill_parts(p, blockIdx.x + 1, x)) {  // grid.x = main_ctas - 1
        return;
    }
    const PrefillUnit unit = x.unit;
    const int         h = x.h, cf = x.cf, cl = x.cl;
    const int G = p.num_heads / p.num_kv_heads, TQ = kPfRows / G;
    const int r = threadIdx.x & 127, tq = r / G, g = r - tq * G;
    if (tq >= TQ || unit.q0 + t * TQ + tq >= unit.q_len) {
        return;
    }
    constexpr int kC = kPfD / 4 / kPfMergeZ / 2;            // groups of four dims per thread
    const int   c0 = (blockIdx.z * 2 + (threadIdx.x >> 7)) * kC;  // the first of them
    const float c  = p.qk_scale;
    float       M = -INFINITY, L = 0.f, o[4 * kC];
#pragma unroll
    for (int i = 0; i < 4 * kC; ++i) o[i] = 0.f;
    constexpr int kBatch = 4;  // parts in flight
    for (int cta = cf; cta <= cl; cta += kBatch) {
        float2 ml[kBatch];
        float4 v[kBatch][kC];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            ml[i] = make_float2(-INFINITY, 0.f);
            if (cta + i <= cl) {
                const float* part = p.partial + ((size_t)x.slot(cta + i) * 2 + t) * kPfPartialFloats;
                ml[i]   = __ldcg(reinterpret_cast<const float2*>(part + (size_t)kPfRows * kPfD) + r);
#pragma unroll
                for (int k = 0; k < kC; ++k) v[i][k] = __ldcg(reinterpret_cast<const float4*>(part) + (c0 + k) * kPfRows + r);
            }
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            if (ml[i].x == -INFINITY) {
                continue;  // no key of the part is visible to the row: its accumulator may not even have been written
            }
            const float m = fmaxf(M, ml[i].x);
            const float a = exp2_approx((M - m) * c), w = exp2_approx((ml[i].x - m) * c);
            M = m;
            L = fmaf(L, a, ml[i].y * w);
#pragma unroll
            for (int k = 0; k < 4 * kC; ++k) o[k] = fmaf(o[k], a, (&v[i][k >> 2].x)[k & 3] * w);
        }
    }
    const float inv = 1.f / L;
    T*          dst = reinterpret_cast<T*>(p.out) + ((size_t)unit.tok0 + unit.q0 + t * TQ + tq) * p.out_stride + ((size_t)h * G + g) * kPfD + c0 * 4;
#pragma unroll
    for (int k = 0; k < 4 * kC; k += 8) {
        uint4 y;
        y.x = Ops::pack2(o[k] * inv, o[k + 1] * inv);
        y.y = Ops::pack2(o[k + 2] * inv, o[k + 3] * inv);
        y.z = Ops::pack2(o[k + 4] * inv, o[k + 5] * inv);
        y.w = Ops::pack2(o[k + 6] * inv, o[k + 7] * inv);
        *reinterpret_cast<uint4*>(dst + k) = y;
    }
}

}  // namespace attn
}  // namespace b200
