// Paged-KV flash-decoding attention for sm_100a (B200).
//
// Replaces, behind the C ABI in include/b200_turbomind.h, the reference's
//   dispatchDecoding<T>(AttentionParams<T>)            src/turbomind/kernels/attention/decoding.cu:13-39
//   attention_kernel<Decoding_MMA<...>>                attention_universal.h:355-553, impl_81616.h
//   attention::reduce / invokeReduceV3                 reduce.cu:13-298
// It is NOT a port: the design is a persistent, warp-specialised kernel
//   * one producer warp streams KV page tiles (64 tokens of one kv-head) from the block table into a
//     shared-memory ring with 1-D TMA bulk copies (cp.async.bulk + mbarrier complete_tx);
//   * four consumer warps de-quantise int8/int4 in registers straight into mma.sync fragments
//     (K as A-operand of S = K.Q^T, V^T as A-operand of O^T = V^T.P), online base-2 softmax;
//   * work is a flat, balanced partition of all (sequence, kv-head, tile) units over a fixed grid
//     ("stream-K"); a segment that straddles CTAs leaves fp32 partials that a fix-up kernel merges in
//     a fixed order (deterministic run to run).
// The kernel is HBM-bound (every KV byte is read exactly once); tensor cores are used only because
// CUDA-core FMA throughput cannot keep up with 6.5 TB/s of int8/int4 operands.
//
// Shared-memory tile layout: rows (tokens) of 128 / 256 bytes are copied in groups of 16 with 32 bytes of padding between
// groups; together with the slot->token permutation below this makes every LDS of the fragment loads
// bank-conflict free without TMA swizzling (pages are addressed by pointer, so no tensor map exists for them).
// Rows of 64 bytes (int4) are copied in two groups of 32 with 64 bytes between them, so that a tile takes few copies: the
// loads of K are free of conflicts, those of V take two passes each.
#pragma once

#include "common.cuh"

namespace b200 {
namespace attn {

constexpr int kHeadDim       = 128;
constexpr int kTile          = 64;  // tokens per pipeline stage
constexpr int kConsumerWarps = 4;
constexpr int kThreads       = (kConsumerWarps + 1) * 32;
constexpr int kMaxGroup      = 8;  // q heads per kv head handled by one CTA (mma N)

template<int KVBITS>
struct TileCfg {
    static constexpr bool kQuant     = KVBITS != 16;
    static constexpr int  kRowBytes  = kHeadDim * KVBITS / 8;
    static constexpr int  kGroupRows = KVBITS == 4 ? 32 : 16;
    static constexpr int  kGroupPad  = KVBITS == 4 ? 64 : 32;
    static constexpr int  kGroupSize = kGroupRows * kRowBytes + kGroupPad;
    // int4: V begins where K ends (no padding behind the last group), as it does in a page of one tile: K's second and V's first half are one copy
    static constexpr int  kTileBytes = (kTile / kGroupRows) * kGroupSize - (KVBITS == 4 ? kGroupPad : 0);
    static constexpr int  kParamBytes = kQuant ? kTile * 4 : 0;  // (scale, zero) as T per token
    static constexpr int  kStageBytes = 2 * kTileBytes + 2 * kParamBytes;
    // offsets inside a stage
    static constexpr int kOffK  = 0;
    static constexpr int kOffV  = kTileBytes;
    static constexpr int kOffKP = 2 * kTileBytes;
    static constexpr int kOffVP = 2 * kTileBytes + kParamBytes;
};

// ------------------------------------------------------------------------------------------------
// RoPE constants: init_rope_kernel_param (src/turbomind/models/attention_weight.cc:37-93)
// ------------------------------------------------------------------------------------------------
struct RopeConst {
    int   type;
    int   dim;
    float scale_factor;
    float inv_factor;
    float attention_scaling;
    float llama3_alpha, llama3_beta;
    float yarn_div2, yarn_mulmin;
    int   exact;  // b200_rope_config::exact_math
};


__device__ __forceinline__ float mul_ftz(float a, float b)
{
    float c;
    asm("mul.ftz.f32 %0, %1, %2;" : "=f"(c) : "f"(a), "f"(b));
    return c;
}
__device__ __forceinline__ float fma_ftz(float a, float b, float c)
{
    float d;
    asm("fma.rn.ftz.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// inv_freq of the pair starting at even dim `idx` (rotary_embedding.h:10-52).
// Default: the instruction sequence of the reference's release build (--use_fast_math: ex2.approx.ftz, ftz
// multiplies, mul+add contracted to fma) so results are bit-identical to TurboMind on the same GPU; `exact`:
// correctly rounded exp2 and un-fused fp32 ops (what the CPU oracle computes).
__device__ __forceinline__ float rope_inv_freq(const RopeConst& r, int idx)
{
    if (r.exact) {
        const float e    = __fmul_rn((float)idx, r.scale_factor);
        const float freq = (float)exp2((double)e);
        if (r.type == 5) {
            float sm = fmaf(r.llama3_alpha, freq, -r.llama3_beta);
            sm       = fmaxf(0.f, fminf(1.f, sm));
            const float a = __fmul_rn(__fsub_rn(1.f, sm), freq);
            const float b = __fmul_rn(a, r.inv_factor);
            const float c = __fmul_rn(sm, freq);
            return __fadd_rn(b, c);
        }
        if (r.type == 4) {
            float alpha = __fsub_rn(__fmul_rn((float)idx, r.yarn_div2), r.yarn_mulmin);
            alpha       = fmaxf(0.f, fminf(1.f, alpha));
            const float t = __fmul_rn(__fmul_rn(freq, alpha), __fsub_rn(1.f, r.inv_factor));
            return __fsub_rn(freq, t);
        }
        return __fmul_rn(r.inv_factor, freq);
    }
    const float freq = exp2_approx(mul_ftz((float)idx, r.scale_factor));
    if (r.type == 5) {
        // (1 - smooth) * freq * inv_factor + smooth * freq
        float sm = fma_ftz(r.llama3_alpha, freq, -r.llama3_beta);
        sm       = fmaxf(0.f, fminf(1.f, sm));
        const float a = mul_ftz(mul_ftz(1.f - sm, freq), r.inv_factor);
        return fma_ftz(sm, freq, a);
    }
    if (r.type == 4) {
        // freq - freq * alpha * (1 - inv_factor)
        float alpha = fma_ftz((float)idx, r.yarn_div2, -r.yarn_mulmin);
        alpha       = fmaxf(0.f, fminf(1.f, alpha));
        const float t = mul_ftz(freq, alpha);
        return fma_ftz(-t, 1.f - r.inv_factor, freq);
    }
    return mul_ftz(r.inv_factor, freq);
}

__device__ __forceinline__ float2 rope_cos_sin(const RopeConst& r, int idx, int pos)
{
    if (r.exact) {
        const float ang = __fmul_rn((float)pos, rope_inv_freq(r, idx));
        double      s, c;
        sincos((double)ang, &s, &c);
        return make_float2(__fmul_rn((float)c, r.attention_scaling), __fmul_rn((float)s, r.attention_scaling));
    }
    // sincosf under --use_fast_math = sin.approx.ftz / cos.approx.ftz of the ftz product (no range reduction)
    const float ang = mul_ftz((float)pos, rope_inv_freq(r, idx));
    float       s, c;
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(ang));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(ang));
    return make_float2(mul_ftz(c, r.attention_scaling), mul_ftz(s, r.attention_scaling));
}


// bias + RoPE of 4 consecutive dims [di, di + 4) of one head vector, T arithmetic as the reference's release build
// (rotary_embedding.h:168-181 compiled with --use_fast_math: `c*x0 - s*x1` as a product and a fused multiply-add)
template<class T>
__device__ __forceinline__ void rope_rotate4(T (&x)[4], const float2 (&cs)[2], const RopeConst& rope, int di)
{
    using Ops = TypeOps<T>;
    if (rope.type == 0) {
        return;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (di + 2 * i < rope.dim) {
            const T c = Ops::from_f32(cs[i].x), s = Ops::from_f32(cs[i].y);
            const T a = x[2 * i], bb = x[2 * i + 1];
            x[2 * i]     = Ops::fma(c, a, Ops::neg(Ops::mul(s, bb)));
            x[2 * i + 1] = Ops::fma(c, bb, Ops::mul(s, a));
        }
    }
}

// out of line: the exact-math variant drags double-precision sincos (and its stack frame) into whoever inlines it
inline __device__ __noinline__ float2 rope_cos_sin_call(const RopeConst& r, int idx, int pos)
{
    return rope_cos_sin(r, idx, pos);
}

// (cos, sin) of the two pairs starting at even dim `di` for position `ti`: from the per-step table when there is one
__device__ __forceinline__ void rope_cs2(float2 (&cs)[2], const RopeConst& rope, const float2* table, int tok, int di, int ti)
{
    if (table) {
        const float4 v = *reinterpret_cast<const float4*>(table + (size_t)tok * (kHeadDim / 2) + (di >> 1));
        cs[0]          = make_float2(v.x, v.y);
        cs[1]          = make_float2(v.z, v.w);
    }
    else {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            cs[i] = (rope.type != 0 && di + 2 * i < rope.dim) ? rope_cos_sin_call(rope, di + 2 * i, ti) : make_float2(1.f, 0.f);
        }
    }
}

template<class T>
__device__ __forceinline__ void load4(const T* p, T (&x)[4])
{
    uint2 u                          = *reinterpret_cast<const uint2*>(p);
    *reinterpret_cast<uint2*>(&x[0]) = u;
}

// Quantise one K or V head vector spread over a warp (lane = 4 consecutive dims): warp_stats + ConvertKvCache
// (quantization.h:341-366, 427-490).  Returns this lane's packed bytes in `bytes` (int8: 4 bytes; int4: the even lane of a pair
// holds 4 bytes covering 8 dims, valid = false on odd lanes) and the (scale, zero) pair as two T in one u32.
template<class T, int KVBITS>
__device__ __forceinline__ void quantize_head(const T (&x)[4], int lane, uint32_t& bytes, bool& valid, uint32_t& param)
{
    using Ops = TypeOps<T>;
    float mn = Ops::to_f32(x[0]), mx = mn;
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        mn = fminf(mn, Ops::to_f32(x[i]));
        mx = fmaxf(mx, Ops::to_f32(x[i]));
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, m));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
    }
    constexpr float inv_q_max = 1.0f / (float)((1 << KVBITS) - 1);
    const T         scale     = Ops::from_f32(__fmul_rn(__fsub_rn(mx, mn), inv_q_max));
    const T         zero      = Ops::from_f32(mn);
    const T         inv_scale = Ops::from_f32(__fdiv_rn(1.f, Ops::to_f32(scale)));
    uint32_t        q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        q[i] = Ops::round_u8(Ops::mul(Ops::sub(x[i], zero), inv_scale));
        if (KVBITS == 4) {
            q[i] = min(q[i], 15u);
        }
    }
    if constexpr (KVBITS == 8) {
        bytes = q[0] | (q[1] << 8) | (q[2] << 16) | (q[3] << 24);
        valid = true;
    }
    else {
        // nibble j of each u32 holds element [0,2,4,6,1,3,5,7][j]  (ConvertKvCache<T,uint4_t>::pack)
        const uint32_t mine = (lane & 1) ? ((q[0] << 8) | (q[2] << 12) | (q[1] << 24) | (q[3] << 28)) :
                                           ((q[0]) | (q[2] << 4) | (q[1] << 16) | (q[3] << 20));
        const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
        bytes = mine | other;
        valid = (lane & 1) == 0;
    }
    T pr[2] = {scale, zero};
    param   = *reinterpret_cast<uint32_t*>(&pr[0]);
}

struct KernelParams {
    const void* q_rot;  // [token][Hq][D]  (bias + RoPE applied)
    void*       out;    // [token][Hq*D], row stride out_stride elements
    int64_t     out_stride;
    char**      block_ptrs;
    const int*  cu_block_nums;  // [B+1]
    const int*  cu_k_len;       // [B+1]
    const int*  tile_prefix;    // [B+1] prefix sum of tiles per sequence (plan kernel)
    float*      partial_O;      // [2*grid][8][128]
    float*      partial_ML;     // [2*grid][8][2]
    int         layer_offset;   // byte offset of this layer inside a block
    int         block_len;
    int         batch;
    int         num_heads;
    int         num_kv_heads;
    float       qk_scale;  // log2(e)/sqrt(D)  (AttentionParams::inv_sqrt_dh)
    int         out_mt;    // > 0: write `out` in the UMMA K-major tile layout [Hq*D/8][out_mt][8]
    // ---- in-kernel prologue (fused & 1): bias + RoPE of q at segment start, and the warp that owns the new token's slot
    // quantises K/V, stores them into the page and patches its shared-memory tile (attention_universal.h:168-348 does the
    // same inside the reference kernel); q_rot is then unused
    int            fused;  // bit 0: in-kernel prologue, bit 1: in-kernel fix-up (the CTA that completes a straddling
                           // (sequence, kv-head) last merges its partials; no reduce kernel)
    const void*    q;
    const void*    k;
    const void*    v;
    int64_t        stride;
    const void*    q_bias;
    const void*    k_bias;
    const void*    v_bias;
    const int*     cu_q_len;
    const int*     readonly_block_num;
    const float2*  rope_table;
    RopeConst      rope;
    int*           seg_counters;  // [grid] arrivals per straddling segment, by the first CTA that has keys of it; zero on entry, left zero
    int            grid_main;
    int            early;  // 1: the producer warp streams KV tiles before griddepcontrol.wait, 2: the consumers look up before it, too (see the kernel's head)
};

// slot (0..15 inside a warp's 16-key MMA) -> token index inside the 64-token tile; slot c + 8 holds the token behind that of slot c
B200_DEVICE int slot_token(int c, int warp)
{
    // group table G = [0,2,1,3,2,0,3,1] packed 2 bits each
    const int grp = (0x72D8 >> (2 * (c & 7))) & 3;
    const int i   = (c >> 3) + 2 * ((c & 7) >> 2);
    return 16 * grp + 4 * warp + i;
}
// the consumer warp whose 16 keys hold a token
B200_DEVICE int token_warp(int tok)
{
    return (tok >> 2) & 3;
}

template<int KVBITS>
B200_DEVICE int token_smem_offset(int tok)
{
    using Cfg = TileCfg<KVBITS>;
    return tok / Cfg::kGroupRows * Cfg::kGroupSize + tok % Cfg::kGroupRows * Cfg::kRowBytes;
}

// first dim of the 4 consecutive dims lane-class t contracts in k-step j of S = K.Q^T
template<int KVBITS>
B200_DEVICE int qk_dim0(int t, int j)
{
    if constexpr (KVBITS == 8) {
        return 16 * t + 64 * (j >> 2) + 4 * (j & 3);
    }
    else if constexpr (KVBITS == 4) {
        return 32 * t + 4 * j;
    }
    else {
        return 8 * (t + 4 * (j >> 1)) + 4 * (j & 1);
    }
}

// output dim held by lane-group g in m-tile j, element e (0: m-slot g, 1: m-slot g+8)
template<int KVBITS>
B200_DEVICE int pv_dim(int g, int j, int e)
{
    if constexpr (KVBITS == 16) {
        return (j < 4 ? 8 * g + 2 * j : 64 + 8 * g + 2 * (j - 4)) + e;
    }
    else {
        return 16 * g + 2 * j + e;
    }
}

struct WorkIter {
    int        batch, hkv;
    const int* prefix;
    int        b, h, tile, tiles;
    B200_DEVICE void seek(long long idx)
    {
        // find b: hkv*prefix[b] <= idx < hkv*prefix[b+1]
        int lo = 0, hi = batch;
        while (hi - lo > 1) {
            int mid = (lo + hi) >> 1;
            if ((long long)hkv * prefix[mid] <= idx) {
                lo = mid;
            }
            else {
                hi = mid;
            }
        }
        b     = lo;
        tiles = prefix[b + 1] - prefix[b];
        // lower_bound above may land on an empty sequence only if idx is past the end
        long long r = idx - (long long)hkv * prefix[b];
        h           = tiles ? (int)(r / tiles) : 0;
        tile        = tiles ? (int)(r % tiles) : 0;
    }
    B200_DEVICE void next()
    {
        if (++tile == tiles) {
            tile = 0;
            if (++h == hkv) {
                h = 0;
                do {
                    ++b;
                    tiles = (b < batch) ? prefix[b + 1] - prefix[b] : 1;
                } while (tiles == 0);
            }
        }
    }
};

// The main-kernel CTAs that hold a piece of segment (sequence b, kv-head h).  CTA c owns units [total * c / grid,
// total * (c + 1) / grid).  With total >= grid every CTA is non-empty and the pieces sit in CTAs cf..cl; with total < grid a
// CTA holds at most ONE unit (= one tile), empty CTAs lie in between, and the pieces are the segment's `tiles` units, unit
// u living in CTA ((u + 1) * grid - 1) / total.  (Walking cf..cl in both cases would read the never-written -- or,
// worse, stale -- partial slots of the empty CTAs in between.)
struct SegCtas {
    int       cf, cl, first_slot, n;  // n = number of pieces
    int       sparse;
    long long s0, total;
};

template<class T, int KVBITS, int STAGES>
struct SharedStorage {
    using Cfg = TileCfg<KVBITS>;
    alignas(128) uint8_t stage[STAGES][Cfg::kStageBytes];
    alignas(16) float merge_O[2][kMaxGroup][kHeadDim];
    float    merge_M[kConsumerWarps][kMaxGroup];
    float    merge_L[kConsumerWarps][kMaxGroup];
    float    final_M[kMaxGroup];
    float    final_L[kMaxGroup];
    SegCtas  seg;       // in-kernel fix-up: where the pieces of the segment being closed live
    int      fix_last;  // ... and whether this CTA arrived last (it merges)
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
};

// swizzled index into the [head][128] fp32 merge rows: keeps (d, d+1) pairs adjacent and spreads the 16 lanes of
// a half-warp over 16 distinct 8-byte slots (bank-conflict-free 64-bit accesses in the segment merge)
B200_DEVICE int merge_idx(int hd, int d)
{
    return hd * kHeadDim + (d ^ ((((d >> 5) & 3) << 1) | ((hd >> 1) << 3)));
}

template<class T, int KVBITS>
struct ConsumerCtx {
    int      warp, g, t;
    // what belongs to slots c + 8 lies a token behind
    int      tokA, tokV0, tokV1;     // keys of row g; of k-slots 2t, 2t + 1
    uint32_t offA, offV0, offV1;     // their rows, this lane's bytes of them included
};

// int8 / int4 pages with f16 activations: the codes enter the tensor cores as they are.  A code in the low mantissa bits of an f16 lane
// IS code * 2^-24 (2^-20 four bits up), a subnormal, so a lane costs one permute or mask instead of permute, subtraction and fma; the
// token's (scale, zero) are applied to the products in fp32:
//   s_t = scale_t * 2^24 * (code_t . q) + zero_t * sum(q);    P_t = exp2(..),   P'_t = T(P_t * scale_t * kappa)
//   kappa * O_d = 2^24 * sum_t P'_t (code_td - mid) + sum_t P'_t * (zero_t / scale_t + mid)
// mid is the middle of the codes: the codes enter as they are, and every kRecentre tiles mid * sum P' is taken off the accumulators.  Left
// in, it makes them a hundred times larger than the output that remains when the zero part is added, and the tensor cores cut a product's
// bits off at the accumulator's last one (64 sequences of 8192 int8 keys: error against 64 bits 5.3e-4 with T-rounded values, 9.9e-4
// without this, 4.5e-4 with it).
// The same rounded P' stands in both sums, so its rounding acts on V as before; K and V are no longer rounded to T.  A warp's 16 keys with
// a scale outside [kMin, kMax] (0 among them: a constant vector) take the T-rounded values as the other types do: inside, scale * kappa
// is at least 1, so that P' is nowhere rounded more coarsely than T(P), and at most 2^15, so that it stays finite (P is 1 at most, but
// for the rounding of the exponent).
// Measured (B200, 32 / 8 heads, whole operator, T-rounded values -> this): int4, 128 x 4096: 190 -> 174 us, error against 64 bits 5.1e-4 ->
// 4.3e-4; int8, 64 x 2048: 62 -> 57 us, 4.9e-4 -> 4.0e-4.
template<class T, int KVBITS>
constexpr bool kCodesInMma = std::is_same<T, half>::value && KVBITS != 16;
template<int KVBITS>
struct CodeScale {
    static constexpr float kappa = KVBITS == 8 ? 65536.f : 16384.f;  // values that span up to 127 (int8: 255 / 2) or 30 (int4: 15 * 2)
    static constexpr float kMin  = 1.f / kappa;
    static constexpr float kMax  = 32768.f / kappa;
    static constexpr float mid   = KVBITS == 8 ? 128.f : 8.f;
    // what one unit of accumulator j (pv_dim) stands for
    B200_DEVICE static float unit(int j) { return KVBITS == 8 || !(j & 1) ? 16777216.f : 1048576.f; }
};
B200_DEVICE float2 half2_to_float2(uint32_t x)
{
    return __half22float2(reinterpret_cast<const half2&>(x));
}

constexpr int kRecentre = 8;  // a multiple of kTilesAtOnce

// Tiles that a consumer warp takes at once: their scores, then their values, are one stretch of code each, so that two chains of products run beside one
// another, and the vote and the loop are paid once; maxima over lanes are taken only where a score lies above them.  A tile is weighed against the maximum
// of the tiles up to it, not of those taken with it, and the sums run in the order of the tiles, so that outputs do not depend on this number.
// int4 pages, 32 / 8 heads, whole operator (us, four sets of pages in turn), with one / two / four at once: 128 x 4096 f16 157 / 144 / 174 (four spill), bf16
// 182 / 164 / 188, 64 x 2048 51.8 / 49.2 / 61, 16 x 100 - 300 15.3 / 15.4 / 16.0 (before tiles took fewer copies: 128 x 4096 175 and 197 in bf16, 64 x 2048 55.3,
// 16 x 100 - 300 16.0).  int8 reads its pages at 6.2 TB/s with one and gains nothing (55 us, 62 with two: only three stages fit).
template<int KVBITS>
constexpr int kTilesAtOnce = KVBITS == 4 ? 2 : 1;

// kCodesInMma: sums that go with the accumulators of a run of tiles (heads 2t, 2t + 1)
struct CodeSums {
    float q[2];  // q's dims
    float a[2];  // this lane's part of sum P' (zero / scale + mid)
    float w[2];  // this lane's part of sum P' since mid was last taken off the accumulators
};

template<int KVBITS>
B200_DEVICE void recentre(float (&O)[8][4], CodeSums& sums)
{
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float w = sums.w[i];
        w += __shfl_xor_sync(0xffffffffu, w, 4);
        w += __shfl_xor_sync(0xffffffffu, w, 8);
        w += __shfl_xor_sync(0xffffffffu, w, 16);
        sums.w[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float f = CodeScale<KVBITS>::mid / CodeScale<KVBITS>::unit(j);
            O[j][i]       = fmaf(-f, w, O[j][i]);
            O[j][i + 2]   = fmaf(-f, w, O[j][i + 2]);
        }
    }
}

// scores of this warp's 16 keys of a tile.  `st` = shared address of the stage.  S[0], S[1]: row g (tokA) heads 2t, 2t + 1;  S[2], S[3]: row g + 8 (tokB)
template<class T, int KVBITS>
B200_DEVICE void score_tile(const ConsumerCtx<T, KVBITS>& cx, uint32_t st, const uint32_t (&qf)[8][2], const CodeSums& sums, float (&S)[4])
{
    using Ops = TypeOps<T>;
    using Cfg = TileCfg<KVBITS>;
    const int t = cx.t;
    const int tokA = cx.tokA, tokB = cx.tokA + 1;
    const uint32_t rowA = st + Cfg::kOffK + cx.offA, rowB = rowA + Cfg::kRowBytes;
    S[0] = S[1] = S[2] = S[3] = 0.f;
    if constexpr (kCodesInMma<T, KVBITS>) {
        const uint2  kp = lds64(st + Cfg::kOffKP + tokA * 4);
        const float2 zA = half2_to_float2(kp.x), zB = half2_to_float2(kp.y);
        if constexpr (KVBITS == 8) {
            uint4 ka[2], kb[2];
            ka[0] = lds128(rowA);
            ka[1] = lds128(rowA + 64);
            kb[0] = lds128(rowB);
            kb[1] = lds128(rowB + 64);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t ua = (&ka[j >> 2].x)[j & 3], ub = (&kb[j >> 2].x)[j & 3];
                const uint32_t a[4] = {__byte_perm(ua, 0u, 0x4140), __byte_perm(ub, 0u, 0x4140), __byte_perm(ua, 0u, 0x4342), __byte_perm(ub, 0u, 0x4342)};
                Ops::mma16816(S, a, qf[j]);
            }
        }
        else {
            // nibbles 0 / 4 and 2 / 6 of a word lie at bit 0 of their lanes (dims 0, 1 | 4, 5), nibbles 1 / 5 and 3 / 7 at bit 4
            // (dims 2, 3 | 6, 7): one product for each kind, with the query's fragments paired alike
            const uint4 ka = lds128(rowA), kb = lds128(rowB);
            float       S4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t ua = (&ka.x)[i], ub = (&kb.x)[i], va = ua >> 8, vb = ub >> 8;
                const uint32_t a0[4] = {ua & 0x000f000fu, ub & 0x000f000fu, va & 0x000f000fu, vb & 0x000f000fu};
                const uint32_t a1[4] = {ua & 0x00f000f0u, ub & 0x00f000f0u, va & 0x00f000f0u, vb & 0x00f000f0u};
                const uint32_t b0[2] = {qf[2 * i][0], qf[2 * i + 1][0]}, b1[2] = {qf[2 * i][1], qf[2 * i + 1][1]};
                Ops::mma16816(S, a0, b0);
                Ops::mma16816(S4, a1, b1);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) S[i] = fmaf(S4[i], 0.0625f, S[i]);
        }
        const float sA = zA.x * 16777216.f, sB = zB.x * 16777216.f;
        S[0] = fmaf(sA, S[0], zA.y * sums.q[0]);
        S[1] = fmaf(sA, S[1], zA.y * sums.q[1]);
        S[2] = fmaf(sB, S[2], zB.y * sums.q[0]);
        S[3] = fmaf(sB, S[3], zB.y * sums.q[1]);
    }
    else if constexpr (KVBITS == 8) {
        const uint32_t pA  = lds32(st + Cfg::kOffKP + tokA * 4);
        const uint32_t pB  = lds32(st + Cfg::kOffKP + tokB * 4);
        const uint32_t sA2 = __byte_perm(pA, pA, 0x1010), zA2 = __byte_perm(pA, pA, 0x3232);
        const uint32_t sB2 = __byte_perm(pB, pB, 0x1010), zB2 = __byte_perm(pB, pB, 0x3232);
        uint4          ka[2], kb[2];
        ka[0] = lds128(rowA);
        ka[1] = lds128(rowA + 64);
        kb[0] = lds128(rowB);
        kb[1] = lds128(rowB + 64);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t ua = (&ka[j >> 2].x)[j & 3];
            const uint32_t ub = (&kb[j >> 2].x)[j & 3];
            uint32_t       a[4];
            Ops::cvt_u8x4(ua, a[0], a[2]);
            Ops::cvt_u8x4(ub, a[1], a[3]);
            a[0] = Ops::fma2(a[0], sA2, zA2);
            a[2] = Ops::fma2(a[2], sA2, zA2);
            a[1] = Ops::fma2(a[1], sB2, zB2);
            a[3] = Ops::fma2(a[3], sB2, zB2);
            Ops::mma16816(S, a, qf[j]);
        }
    }
    else if constexpr (KVBITS == 4) {
        const uint32_t pA  = lds32(st + Cfg::kOffKP + tokA * 4);
        const uint32_t pB  = lds32(st + Cfg::kOffKP + tokB * 4);
        const uint32_t sA2 = __byte_perm(pA, pA, 0x1010), zA2 = __byte_perm(pA, pA, 0x3232);
        const uint32_t sB2 = __byte_perm(pB, pB, 0x1010), zB2 = __byte_perm(pB, pB, 0x3232);
        const uint4    ka  = lds128(rowA);
        const uint4    kb  = lds128(rowB);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t ha[4], hb[4];
            Ops::cvt_u4x8((&ka.x)[i], ha);
            Ops::cvt_u4x8((&kb.x)[i], hb);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                ha[x] = Ops::fma2(ha[x], sA2, zA2);
                hb[x] = Ops::fma2(hb[x], sB2, zB2);
            }
            // u32 i covers dims 8i..8i+7 of this lane's chunk: k-steps 2i (dims 0-3) and 2i+1 (dims 4-7)
            uint32_t a0[4] = {ha[0], hb[0], ha[1], hb[1]};
            uint32_t a1[4] = {ha[2], hb[2], ha[3], hb[3]};
            Ops::mma16816(S, a0, qf[2 * i]);
            Ops::mma16816(S, a1, qf[2 * i + 1]);
        }
    }
    else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 ka = lds128(rowA + 64 * i);
            const uint4 kb = lds128(rowB + 64 * i);
            uint32_t    a0[4] = {ka.x, kb.x, ka.y, kb.y};
            uint32_t    a1[4] = {ka.z, kb.z, ka.w, kb.w};
            Ops::mma16816(S, a0, qf[2 * i]);
            Ops::mma16816(S, a1, qf[2 * i + 1]);
        }
    }
}

// the maxima (over all lanes of a head) grow to at least mx: what was accumulated against the former ones is rescaled
template<class T, int KVBITS>
B200_DEVICE void grow_maxima(const float (&mx)[2], float c, float (&O)[8][4], float (&M)[2], float (&L)[2], CodeSums& sums)
{
    float newM[2] = {fmaxf(M[0], mx[0]), fmaxf(M[1], mx[1])};
    // a whole 16-key slice can only be fully masked in a residue tile
    const bool dead0 = newM[0] == -INFINITY, dead1 = newM[1] == -INFINITY;
    if (newM[0] != M[0] || newM[1] != M[1]) {
        const float r0 = dead0 ? 1.f : exp2_approx((M[0] - newM[0]) * c);
        const float r1 = dead1 ? 1.f : exp2_approx((M[1] - newM[1]) * c);
        L[0] *= r0;
        L[1] *= r1;
        if constexpr (kCodesInMma<T, KVBITS>) {
            sums.a[0] *= r0, sums.w[0] *= r0;
            sums.a[1] *= r1, sums.w[1] *= r1;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            O[j][0] *= r0;
            O[j][1] *= r1;
            O[j][2] *= r0;
            O[j][3] *= r1;
        }
        M[0] = newM[0];
        M[1] = newM[1];
    }
}

// P = exp2(c S - mc)
B200_DEVICE void weights(const float (&S)[4], float c, float mc0, float mc1, float (&P)[4], float (&L)[2])
{
    P[0] = exp2_approx(fmaf(S[0], c, -mc0));
    P[1] = exp2_approx(fmaf(S[1], c, -mc1));
    P[2] = exp2_approx(fmaf(S[2], c, -mc0));
    P[3] = exp2_approx(fmaf(S[3], c, -mc1));
    L[0] += P[0] + P[2];  // per-lane partial row sums; reduced across g at segment end
    L[1] += P[1] + P[3];
}

template<class T, int KVBITS>
struct ValueRows {
    uint32_t row0, row1, row2, row3;  // of k-slots 2t, 2t + 1, 2t + 8, 2t + 9
    B200_DEVICE ValueRows(const ConsumerCtx<T, KVBITS>& cx, uint32_t st)
    {
        constexpr int next = TileCfg<KVBITS>::kRowBytes;
        row0 = st + TileCfg<KVBITS>::kOffV + cx.offV0, row1 = st + TileCfg<KVBITS>::kOffV + cx.offV1;
        row2 = row0 + next, row3 = row1 + next;
    }
};

// (scale, zero) of this lane's two values
struct ValueParams {
    float2 A, B;
};
template<class T, int KVBITS>
B200_DEVICE ValueParams value_params(const ConsumerCtx<T, KVBITS>& cx, uint32_t st)
{
    const uint2 vp = lds64(st + TileCfg<KVBITS>::kOffVP + cx.tokA * 4);
    return {half2_to_float2(vp.x), half2_to_float2(vp.y)};
}
// the values' codes may go into the product as they are
template<int KVBITS>
B200_DEVICE bool fit(const ValueParams& v)
{
    using CS = CodeScale<KVBITS>;
    return v.A.x >= CS::kMin && v.A.x <= CS::kMax && v.B.x >= CS::kMin && v.B.x <= CS::kMax;
}

// O^T += V^T . P of this warp's 16 keys of a tile over the values' codes
template<class T, int KVBITS>
B200_DEVICE void weigh_codes(const ConsumerCtx<T, KVBITS>& cx, uint32_t st, const ValueParams& v, const float (&P)[4], float (&O)[8][4], CodeSums& sums)
{
    using Ops = TypeOps<T>;
    using CS  = CodeScale<KVBITS>;
    const auto [row0, row1, row2, row3] = ValueRows<T, KVBITS>(cx, st);
    const float    kA = v.A.x * CS::kappa, kB = v.B.x * CS::kappa;
    const uint32_t wA = Ops::pack2(P[0] * kA, P[1] * kA), wB = Ops::pack2(P[2] * kB, P[3] * kB);
    const float    rA = __fdividef(v.A.y, v.A.x) + CS::mid, rB = __fdividef(v.B.y, v.B.x) + CS::mid;
    const float2   fA = half2_to_float2(wA), fB = half2_to_float2(wB);
    sums.a[0] = fmaf(fA.x, rA, fmaf(fB.x, rB, sums.a[0]));
    sums.a[1] = fmaf(fA.y, rA, fmaf(fB.y, rB, sums.a[1]));
    sums.w[0] += fA.x + fB.x;
    sums.w[1] += fA.y + fB.y;
    const uint32_t pf[2] = {transpose_8x8_b16(wA), transpose_8x8_b16(wB)};
    if constexpr (KVBITS == 8) {
        const uint4 v0 = lds128(row0), v1 = lds128(row1);
        const uint4 v2 = lds128(row2), v3 = lds128(row3);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            const uint32_t A0 = (&v0.x)[jj], B0 = (&v1.x)[jj], C0 = (&v2.x)[jj], D0 = (&v3.x)[jj];
            const uint32_t X = __byte_perm(A0, B0, 0x5140), Y = __byte_perm(A0, B0, 0x7362);
            const uint32_t X2 = __byte_perm(C0, D0, 0x5140), Y2 = __byte_perm(C0, D0, 0x7362);
            const uint32_t a0[4] = {__byte_perm(X, 0u, 0x4140), __byte_perm(X, 0u, 0x4342), __byte_perm(X2, 0u, 0x4140), __byte_perm(X2, 0u, 0x4342)};
            const uint32_t a1[4] = {__byte_perm(Y, 0u, 0x4140), __byte_perm(Y, 0u, 0x4342), __byte_perm(Y2, 0u, 0x4140), __byte_perm(Y2, 0u, 0x4342)};
            Ops::mma16816(O[2 * jj], a0, pf);
            Ops::mma16816(O[2 * jj + 1], a1, pf);
        }
    }
    else {
        const uint2 v0 = lds64(row0), v1 = lds64(row1);
        const uint2 v2 = lds64(row2), v3 = lds64(row3);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint32_t A0 = (&v0.x)[m], B0 = (&v1.x)[m], C0 = (&v2.x)[m], D0 = (&v3.x)[m];
            const uint32_t Ye = __byte_perm(A0, B0, 0x5410), Yo = __byte_perm(A0, B0, 0x7632);
            const uint32_t Ze = __byte_perm(C0, D0, 0x5410), Zo = __byte_perm(C0, D0, 0x7632);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const uint32_t mask = x & 1 ? 0x00f000f0u : 0x000f000fu;
                const int      sh   = x & 2 ? 8 : 0;
                const uint32_t a[4] = {(Ye >> sh) & mask, (Yo >> sh) & mask, (Ze >> sh) & mask, (Zo >> sh) & mask};
                Ops::mma16816(O[4 * m + x], a, pf);
            }
        }
    }
}

// ... over values rounded to T; beside codes: in the codes' units
template<class T, int KVBITS>
B200_DEVICE void weigh_rounded(const ConsumerCtx<T, KVBITS>& cx, uint32_t st, bool residue, int k_len, int t0, const float (&P)[4], float (&O)[8][4])
{
    using Ops = TypeOps<T>;
    using Cfg = TileCfg<KVBITS>;
    const int  tokV0 = cx.tokV0, tokV1 = cx.tokV1, tokV2 = cx.tokV0 + 1, tokV3 = cx.tokV1 + 1;
    const auto [row0, row1, row2, row3] = ValueRows<T, KVBITS>(cx, st);
    uint32_t pf[2];
    pf[0] = transpose_8x8_b16(Ops::pack2(P[0], P[1]));  // k-slots 2t,2t+1 ; head g
    pf[1] = transpose_8x8_b16(Ops::pack2(P[2], P[3]));  // k-slots 2t+8,2t+9 ; head g
    auto add_rounded = [&](int j, const uint32_t(&a)[4]) {
        if constexpr (kCodesInMma<T, KVBITS>) {
            float d[4] = {0.f, 0.f, 0.f, 0.f};
            Ops::mma16816(d, a, pf);
            const float f = CodeScale<KVBITS>::kappa / CodeScale<KVBITS>::unit(j);
#pragma unroll
            for (int i = 0; i < 4; ++i) O[j][i] = fmaf(d[i], f, O[j][i]);
        }
        else {
            Ops::mma16816(O[j], a, pf);
        }
    };
    if constexpr (KVBITS == 8) {
        uint32_t p0 = lds32(st + Cfg::kOffVP + tokV0 * 4), p1 = lds32(st + Cfg::kOffVP + tokV1 * 4);
        uint32_t p2 = lds32(st + Cfg::kOffVP + tokV2 * 4), p3 = lds32(st + Cfg::kOffVP + tokV3 * 4);
        if (residue) {
            if (t0 + tokV0 >= k_len) p0 = 0;
            if (t0 + tokV1 >= k_len) p1 = 0;
            if (t0 + tokV2 >= k_len) p2 = 0;
            if (t0 + tokV3 >= k_len) p3 = 0;
        }
        const uint32_t s01 = __byte_perm(p0, p1, 0x5410), z01 = __byte_perm(p0, p1, 0x7632);
        const uint32_t s23 = __byte_perm(p2, p3, 0x5410), z23 = __byte_perm(p2, p3, 0x7632);
        const uint4    v0 = lds128(row0), v1 = lds128(row1);
        const uint4    v2 = lds128(row2), v3 = lds128(row3);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            const uint32_t A = (&v0.x)[jj], Bq = (&v1.x)[jj], C = (&v2.x)[jj], Dq = (&v3.x)[jj];
            const uint32_t X = __byte_perm(A, Bq, 0x5140), Y = __byte_perm(A, Bq, 0x7362);
            const uint32_t X2 = __byte_perm(C, Dq, 0x5140), Y2 = __byte_perm(C, Dq, 0x7362);
            uint32_t       a[4];
            Ops::cvt_u8x4(X, a[0], a[1]);
            Ops::cvt_u8x4(X2, a[2], a[3]);
            a[0] = Ops::fma2(a[0], s01, z01);
            a[1] = Ops::fma2(a[1], s01, z01);
            a[2] = Ops::fma2(a[2], s23, z23);
            a[3] = Ops::fma2(a[3], s23, z23);
            add_rounded(2 * jj, a);
            Ops::cvt_u8x4(Y, a[0], a[1]);
            Ops::cvt_u8x4(Y2, a[2], a[3]);
            a[0] = Ops::fma2(a[0], s01, z01);
            a[1] = Ops::fma2(a[1], s01, z01);
            a[2] = Ops::fma2(a[2], s23, z23);
            a[3] = Ops::fma2(a[3], s23, z23);
            add_rounded(2 * jj + 1, a);
        }
    }
    else if constexpr (KVBITS == 4) {
        uint32_t p0 = lds32(st + Cfg::kOffVP + tokV0 * 4), p1 = lds32(st + Cfg::kOffVP + tokV1 * 4);
        uint32_t p2 = lds32(st + Cfg::kOffVP + tokV2 * 4), p3 = lds32(st + Cfg::kOffVP + tokV3 * 4);
        if (residue) {
            if (t0 + tokV0 >= k_len) p0 = 0;
            if (t0 + tokV1 >= k_len) p1 = 0;
            if (t0 + tokV2 >= k_len) p2 = 0;
            if (t0 + tokV3 >= k_len) p3 = 0;
        }
        const uint32_t s01 = __byte_perm(p0, p1, 0x5410), z01 = __byte_perm(p0, p1, 0x7632);
        const uint32_t s23 = __byte_perm(p2, p3, 0x5410), z23 = __byte_perm(p2, p3, 0x7632);
        const uint2    v0 = lds64(row0), v1 = lds64(row1);
        const uint2    v2 = lds64(row2), v3 = lds64(row3);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint32_t A = (&v0.x)[m], Bq = (&v1.x)[m], C = (&v2.x)[m], Dq = (&v3.x)[m];
            // lo16 of a word: elements e0,e2,e4,e6 (nibbles 0-3); hi16: e1,e3,e5,e7
            const uint32_t Ye = __byte_perm(A, Bq, 0x5410), Yo = __byte_perm(A, Bq, 0x7632);
            const uint32_t Ze = __byte_perm(C, Dq, 0x5410), Zo = __byte_perm(C, Dq, 0x7632);
            uint32_t       he[4], ho[4], ge[4], go[4];
            Ops::cvt_u4x8(Ye, he);  // he[x] = (A.e(2x), B.e(2x))   [(n0,n4),(n1,n5),..] of Ye
            Ops::cvt_u4x8(Yo, ho);  // ho[x] = (A.e(2x+1), B.e(2x+1))
            Ops::cvt_u4x8(Ze, ge);
            Ops::cvt_u4x8(Zo, go);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                // element index inside the word: even -> 2x (m-slot g), odd -> 2x+1 (m-slot g+8)
                uint32_t a[4];
                a[0] = Ops::fma2(he[x], s01, z01);
                a[1] = Ops::fma2(ho[x], s01, z01);
                a[2] = Ops::fma2(ge[x], s23, z23);
                a[3] = Ops::fma2(go[x], s23, z23);
                add_rounded(4 * m + x, a);
            }
        }
    }
    else {
        uint4 va[2], vb[2], vc[2], vd[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            va[i] = lds128(row0 + 128 * i);
            vb[i] = lds128(row1 + 128 * i);
            vc[i] = lds128(row2 + 128 * i);
            vd[i] = lds128(row3 + 128 * i);
        }
        if (residue) {
            const uint4 z = make_uint4(0, 0, 0, 0);
            if (t0 + tokV0 >= k_len) va[0] = va[1] = z;
            if (t0 + tokV1 >= k_len) vb[0] = vb[1] = z;
            if (t0 + tokV2 >= k_len) vc[0] = vc[1] = z;
            if (t0 + tokV3 >= k_len) vd[0] = vd[1] = z;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t A = (&va[j >> 2].x)[j & 3], Bq = (&vb[j >> 2].x)[j & 3];
            const uint32_t C = (&vc[j >> 2].x)[j & 3], Dq = (&vd[j >> 2].x)[j & 3];
            uint32_t       a[4];
            a[0] = __byte_perm(A, Bq, 0x5410);  // (dim 2j, keys 2t,2t+1)
            a[1] = __byte_perm(A, Bq, 0x7632);  // (dim 2j+1, ...)
            a[2] = __byte_perm(C, Dq, 0x5410);
            a[3] = __byte_perm(C, Dq, 0x7632);
            Ops::mma16816(O[j], a, pf);
        }
    }

}

// this warp's 16 keys of a tile with the maxima they got; a lane's two keys seen or not
template<class T, int KVBITS>
B200_DEVICE void weigh_tile(const ConsumerCtx<T, KVBITS>& cx, uint32_t st, bool residue, int k_len, int t0, const float (&P)[4], float (&O)[8][4], CodeSums& sums)
{
    if constexpr (kCodesInMma<T, KVBITS>) {
        ValueParams v = value_params<T, KVBITS>(cx, st);
        if (residue && t0 + cx.tokA >= k_len) {
            v.A = make_float2(CodeScale<KVBITS>::kMin, 0.f);
        }
        if (residue && t0 + cx.tokA + 1 >= k_len) {
            v.B = make_float2(CodeScale<KVBITS>::kMin, 0.f);
        }
        if (__all_sync(0xffffffffu, fit<KVBITS>(v))) {
            weigh_codes<T, KVBITS>(cx, st, v, P, O, sums);
            return;
        }
    }
    weigh_rounded<T, KVBITS>(cx, st, residue, k_len, t0, P, O);
}

B200_DEVICE void warp_maxima(float (&mx)[2])
{
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 4));
        mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 8));
        mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 16));
    }
}

// one 64-token tile
template<class T, int KVBITS>
B200_DEVICE void process_tile(const ConsumerCtx<T, KVBITS>& cx, uint32_t st, bool residue, int k_len, int t0, float c,
                              const uint32_t (&qf)[8][2], float (&O)[8][4], float (&M)[2], float (&L)[2], CodeSums& sums)
{
    float S[4];
    score_tile<T, KVBITS>(cx, st, qf, sums, S);
    if (residue && (t0 + cx.tokA >= k_len)) {
        S[0] = S[1] = -INFINITY;
    }
    if (residue && (t0 + cx.tokA + 1 >= k_len)) {
        S[2] = S[3] = -INFINITY;
    }
    float mx[2] = {fmaxf(S[0], S[2]), fmaxf(S[1], S[3])};
    warp_maxima(mx);
    grow_maxima<T, KVBITS>(mx, c, O, M, L, sums);
    const float mc0 = M[0] == -INFINITY ? 0.f : M[0] * c, mc1 = M[1] == -INFINITY ? 0.f : M[1] * c;
    float       P[4];
    weights(S, c, mc0, mc1, P, L);
    weigh_tile<T, KVBITS>(cx, st, residue, k_len, t0, P, O, sums);
}

// NT tiles, all keys of which are seen, as process_tile would take them one after the other: `st` = shared addresses of their stages
template<class T, int KVBITS, int NT>
B200_DEVICE void process_tiles(const ConsumerCtx<T, KVBITS>& cx, const uint32_t (&st)[NT], float c, const uint32_t (&qf)[8][2], float (&O)[8][4],
                               float (&M)[2], float (&L)[2], CodeSums& sums)
{
    float S[NT][4], mx[NT][2];
    bool  grow = false;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        score_tile<T, KVBITS>(cx, st[i], qf, sums, S[i]);
        mx[i][0] = fmaxf(S[i][0], S[i][2]), mx[i][1] = fmaxf(S[i][1], S[i][3]);
        grow = grow || mx[i][0] > M[0] || mx[i][1] > M[1];
    }
    grow = __any_sync(0xffffffffu, grow);
    if (grow) {
#pragma unroll
        for (int i = 0; i < NT; ++i) warp_maxima(mx[i]);
    }
    auto weights_of = [&](int i, float (&P)[4]) {
        if (grow) {
            grow_maxima<T, KVBITS>(mx[i], c, O, M, L, sums);
        }
        const float mc0 = M[0] == -INFINITY ? 0.f : M[0] * c, mc1 = M[1] == -INFINITY ? 0.f : M[1] * c;
        weights(S[i], c, mc0, mc1, P, L);
    };
    if constexpr (kCodesInMma<T, KVBITS>) {
        uint2 raw[NT];
        bool  ok = true;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            raw[i] = lds64(st[i] + TileCfg<KVBITS>::kOffVP + cx.tokA * 4);
            ok     = ok && fit<KVBITS>(ValueParams{half2_to_float2(raw[i].x), half2_to_float2(raw[i].y)});
        }
        if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                float P[4];
                weights_of(i, P);
                weigh_codes<T, KVBITS>(cx, st[i], ValueParams{half2_to_float2(raw[i].x), half2_to_float2(raw[i].y)}, P, O, sums);
            }
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        float P[4];
        weights_of(i, P);
        weigh_tile<T, KVBITS>(cx, st[i], false, 0, 0, P, O, sums);
    }
}

B200_DEVICE void sts32(uint32_t addr, uint32_t v)
{
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
B200_DEVICE void sts64(uint32_t addr, uint2 v)
{
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}

// In-kernel prologue for the new token of (sequence b, kv-head h) at cache position ti (= tile slot `pos`): one warp,
// lane = 4 consecutive dims (the mapping of kv_prologue_kernel, whose arithmetic this repeats instruction for instruction).
template<class T, int KVBITS>
__device__ __noinline__ void new_token_kv(const KernelParams& p, int b, int h, int ti, int pos, int lane, uint32_t st)
{
    using Ops = TypeOps<T>;
    using Cfg = TileCfg<KVBITS>;
    const int ro_len = p.readonly_block_num ? p.readonly_block_num[b] * p.block_len : 0;
    if (ti < ro_len) {
        return;  // inside a shared read-only prefix block: the page already holds this position
    }
    const int tok = p.cu_q_len ? p.cu_q_len[b] : b;
    const int di  = lane * 4;
    T         xk[4], xv[4];
    load4(reinterpret_cast<const T*>(p.k) + (size_t)tok * p.stride + (size_t)h * kHeadDim + di, xk);
    load4(reinterpret_cast<const T*>(p.v) + (size_t)tok * p.stride + (size_t)h * kHeadDim + di, xv);
    if (p.k_bias) {
        T bk[4], bv[4];
        load4(reinterpret_cast<const T*>(p.k_bias) + (size_t)h * kHeadDim + di, bk);
        load4(reinterpret_cast<const T*>(p.v_bias) + (size_t)h * kHeadDim + di, bv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xk[i] = Ops::add(xk[i], bk[i]);
            xv[i] = Ops::add(xv[i], bv[i]);
        }
    }
    float2 cs[2];
    rope_cs2(cs, p.rope, p.rope_table, tok, di, ti);
    rope_rotate4<T>(xk, cs, p.rope, di);

    constexpr int kRow          = Cfg::kRowBytes;
    const int     head_data_sz  = p.block_len * kRow;
    const int     head_param_sz = p.block_len * 4;
    char*         blk = p.block_ptrs[p.cu_block_nums[b] + ti / p.block_len] + p.layer_offset;
    const int     bt  = ti % p.block_len;
    char*         kd  = blk + (size_t)(h * 2) * head_data_sz + (size_t)bt * kRow;
    char*         vd  = kd + head_data_sz;
    const uint32_t srow = token_smem_offset<KVBITS>(pos);
    if constexpr (KVBITS == 16) {
        const uint2 uk = *reinterpret_cast<uint2*>(&xk[0]), uv = *reinterpret_cast<uint2*>(&xv[0]);
        *reinterpret_cast<uint2*>(kd + 8 * lane) = uk;
        *reinterpret_cast<uint2*>(vd + 8 * lane) = uv;
        sts64(st + Cfg::kOffK + srow + 8 * lane, uk);
        sts64(st + Cfg::kOffV + srow + 8 * lane, uv);
    }
    else {
        char* kp = blk + (size_t)p.num_kv_heads * 2 * head_data_sz + (size_t)(h * 2) * head_param_sz + (size_t)bt * 4;
        char* vp = kp + head_param_sz;
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
            uint32_t bytes, param;
            bool     valid;
            quantize_head<T, KVBITS>(kv ? xv : xk, lane, bytes, valid, param);
            char*          dd   = kv ? vd : kd;
            const uint32_t sdat = st + (kv ? Cfg::kOffV : Cfg::kOffK) + srow;
            if constexpr (KVBITS == 8) {
                *reinterpret_cast<uint32_t*>(dd + 4 * lane) = bytes;
                sts32(sdat + 4 * lane, bytes);
            }
            else if (valid) {
                *reinterpret_cast<uint32_t*>(dd + 4 * (lane >> 1)) = bytes;
                sts32(sdat + 4 * (lane >> 1), bytes);
            }
            if (lane == 0) {
                *reinterpret_cast<uint32_t*>(kv ? vp : kp) = param;
                sts32(st + (kv ? Cfg::kOffVP : Cfg::kOffKP) + pos * 4, param);
            }
        }
    }
}

B200_DEVICE SegCtas segment_ctas(const KernelParams& p, int b, int h, int grid_main)
{
    SegCtas         s;
    const int       Hkv   = p.num_kv_heads;
    const int       tiles = p.tile_prefix[b + 1] - p.tile_prefix[b];
    s.total               = (long long)p.tile_prefix[p.batch] * Hkv;
    s.s0                  = (long long)Hkv * p.tile_prefix[b] + (long long)h * tiles;
    const long long s1    = s.s0 + tiles;
    s.cf                  = (int)(((s.s0 + 1) * grid_main - 1) / s.total);
    s.cl                  = (int)((s1 * grid_main - 1) / s.total);
    s.first_slot          = (s.total * s.cf / grid_main != s.s0) ? 1 : 0;
    s.sparse              = s.total < grid_main;
    s.n                   = s.sparse ? tiles : s.cl - s.cf + 1;
    return s;
}

// Merge of the partials of one segment.  Same math as attention::reduce (reduce.cu:90-153): O = sum_k w_k O_k / sum_k w_k L_k,
// w_k = exp2((M_k - M) * c), pieces visited in ascending CTA order whoever runs the merge (deterministic).  Loads bypass L1
// (ld.global.cg): the partials may have been written by other SMs during this very kernel.
template<class T>
__device__ __noinline__ void merge_segment(const KernelParams& p, int b, int h, const SegCtas& sg, int grid_main, int tid,
                                           int nthreads)
{
    using Ops     = TypeOps<T>;
    const int   G = p.num_heads / p.num_kv_heads;
    const float c = p.qk_scale;
    auto slot_of  = [&](int k) {
        if (sg.sparse) {
            return 2 * (int)(((sg.s0 + k + 1) * grid_main - 1) / sg.total);  // one unit per CTA: always its first slot
        }
        const int cta = sg.cf + k;
        return 2 * cta + (k == 0 ? sg.first_slot : 0);
    };
    // thread -> 4 consecutive dims of one head (float4 partial loads)
    for (int i4 = tid; i4 < G * kHeadDim / 4; i4 += nthreads) {
        const int i  = i4 * 4;
        const int hd = i / kHeadDim;
        float     m  = -INFINITY;
        // kBatch pieces' loads in flight, summed in order (one dependent load after the other: 43 us for 27, 3 sequences of 37 - 7001 bf16
        // tokens, 48 / 8 heads, whole operator)
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float  l   = 0.f;
        auto   sum = [&](auto batch) {
            constexpr int kBatch = decltype(batch)::value;
            for (int k0 = 0; k0 < sg.n; k0 += kBatch) {
                float x[kBatch];
    #pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    x[k] = k0 + k < sg.n ? __ldcg(&p.partial_ML[((size_t)slot_of(k0 + k) * kMaxGroup + hd) * 2]) : -INFINITY;
                }
    #pragma unroll
                for (int k = 0; k < kBatch; ++k) m = fmaxf(m, x[k]);
            }
            for (int k0 = 0; k0 < sg.n; k0 += kBatch) {
                float2 ml[kBatch];
                float4 o[kBatch];
    #pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    ml[k] = make_float2(-INFINITY, 0.f);
                    o[k]  = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (k0 + k < sg.n) {
                        const int slot = slot_of(k0 + k);
                        ml[k] = __ldcg(reinterpret_cast<const float2*>(&p.partial_ML[((size_t)slot * kMaxGroup + hd) * 2]));
                        o[k]  = __ldcg(reinterpret_cast<const float4*>(&p.partial_O[(size_t)slot * kMaxGroup * kHeadDim + i]));
                    }
                }
    #pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const float w = (ml[k].x == -INFINITY) ? 0.f : exp2_approx((ml[k].x - m) * c);
                    l += w * ml[k].y;
                    acc.x += w * o[k].x, acc.y += w * o[k].y, acc.z += w * o[k].z, acc.w += w * o[k].w;
                }
            }
        };
        if (sg.n <= 4) {
            sum(std::integral_constant<int, 2>{});  // the usual case of a full batch: two or three pieces
        }
        else {
            sum(std::integral_constant<int, 8>{});
        }
        const int col = h * G * kHeadDim + i;
        T*        dst = reinterpret_cast<T*>(p.out)
                 + (p.out_mt > 0 ? ((size_t)(col >> 3) * p.out_mt + b) * 8 + (col & 7) : (size_t)b * p.out_stride + col);
        uint2 v;
        v.x = Ops::pack2(acc.x / l, acc.y / l);
        v.y = Ops::pack2(acc.z / l, acc.w / l);
        *reinterpret_cast<uint2*>(dst) = v;
    }
}

B200_DEVICE int atom_add_acq_rel_gpu(int* p, int v)
{
    int old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

struct TileDesc {
    const char* blk;  // block base + layer offset
    int         h;
    int         bt;    // token offset of the tile inside the block
    int         rows;  // valid tokens in the tile
};

// Resident CTAs per SM the register budget must allow (the shared-memory ring is sized for the same numbers): the tile
// loop keeps ~125 registers live; the rare paths (new token's K/V, segment merge) are out-of-line calls so they cannot
// inflate it.  __grid_constant__: those calls take the parameter block by reference without a local copy.
template<int KVBITS>
constexpr int min_ctas_per_sm()
{
    return KVBITS == 16 ? 2 : 3;
}

template<class T, int KVBITS, int STAGES>
__global__ void __launch_bounds__(kThreads, min_ctas_per_sm<KVBITS>()) decode_attention_kernel(const __grid_constant__ KernelParams p)
{
    using Ops = TypeOps<T>;
    using Cfg = TileCfg<KVBITS>;
    using SS  = SharedStorage<T, KVBITS, STAGES>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    SS&                                      ss = *reinterpret_cast<SS*>(smem_raw);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // q and the page of the new token come from the prologue kernel right before this one; the tile plan, the block table and
    // the lengths from kernels (or copies) several launches back.  p.early (the caller supplied the plan and the prologue kernel
    // triggers its dependents only AFTER its own griddepcontrol.wait, so everything older than the prologue is complete when
    // this grid starts): the producer warp does not wait here -- it fills the ring with tiles the prologue does not touch
    // (every tile but the last of a sequence) while the prologue runs, and waits before the first tile that holds a new token.
    // p.early == 2: nor do the consumers, which look up their first segment meanwhile and wait before they read q.
    pdl_launch_dependents();
    const bool early = p.early > (warp == kConsumerWarps ? 0 : 1);
    if (!early) {
        pdl_wait();
    }

    const int       Hkv   = p.num_kv_heads;
    const int       G     = p.num_heads / Hkv;
    const long long total = (long long)p.tile_prefix[p.batch] * Hkv;
    const long long lo    = total * blockIdx.x / gridDim.x;
    const long long hi    = total * (blockIdx.x + 1) / gridDim.x;

    // the producer warp owns the ring's barriers: it initialises them and ARRIVES on named barrier 3; the consumers sync on it
    if (warp == kConsumerWarps) {
        if (lane == 0) {
            for (int s = 0; s < STAGES; ++s) {
                mbar_init(smem_u32(&ss.full[s]), 1);
                mbar_init(smem_u32(&ss.empty[s]), kConsumerWarps);
            }
            fence_mbar_init();
        }
        __syncwarp();
        named_bar_arrive(3, kThreads);
    }
    else {
        named_bar_sync(3, kThreads);
    }

    if (lo >= hi) {
        return;
    }

    const uint32_t full0  = smem_u32(&ss.full[0]);
    const uint32_t empty0 = smem_u32(&ss.empty[0]);
    const uint32_t stage0 = smem_u32(&ss.stage[0][0]);

    if (warp == kConsumerWarps) {
        // ================================ producer warp ================================
        // Tile descriptors (block pointer through the block table, valid rows) are fetched 32 at a time, one per
        // lane, one batch AHEAD of the copies being issued, so the dependent global loads
        // (cu_k_len -> cu_block_nums -> block_ptrs) never sit on the critical path of the TMA issue loop.
        const uint64_t policy         = make_evict_first_policy();
        const int      head_data_size = p.block_len * Cfg::kRowBytes;
        const int      head_param_sz  = p.block_len * 4;
        auto           fetch          = [&](long long base) {
            TileDesc        d{nullptr, 0, 0, 0};
            const long long idx = base + lane;
            if (idx < hi) {
                WorkIter it{p.batch, Hkv, p.tile_prefix};
                it.seek(idx);
                const int k_len = p.cu_k_len[it.b + 1] - p.cu_k_len[it.b];
                const int t0    = it.tile * kTile;
                d.rows          = min(kTile, k_len - t0) | (t0 + kTile >= k_len ? 128 : 0);  // bit 7: holds the new token
                d.h             = it.h;
                d.bt            = t0 % p.block_len;
                d.blk           = p.block_ptrs[p.cu_block_nums[it.b] + t0 / p.block_len] + p.layer_offset;
            }
            return d;
        };
        int      s  = 0;
        uint32_t ph = 0;
        bool     pending = early;  // griddepcontrol.wait still to come
        int      issued  = 0;
        TileDesc cur = fetch(lo);
        // Copy roles: lanes 0-7 move the four 16-row groups of K (even) and V (odd), lanes 8/9 the K/V quant params.
        // The ten copies of one tile are issued by ten lanes in ONE pass (a single lane issuing them serially costs
        // ~280 issue slots per tile on the scheduler this warp shares with a consumer warp).
        const int  my_gq    = (lane >> 1) & 3;
        const bool my_v     = lane & 1;
        const bool my_data  = lane < 8;
        const bool my_param = Cfg::kQuant && (lane == 8 || lane == 9);
        for (long long base = lo; base < hi; base += 32) {
            const TileDesc nxt = fetch(base + 32);
            const int      cnt = (int)min((long long)32, hi - base);
            if constexpr (KVBITS == 4) {
                // The lane that holds a tile's descriptor issues its copies: four of them where a page is one tile long, up to six otherwise.  A bulk
                // copy takes its operands from uniform registers, so that lanes which issue together are served one after the other: ten copies per
                // tile cost this warp some 450 issue slots and up to 1290 cycles (consumers that only wait and release: 110 us for 128 x 4096 int4
                // keys, whose bytes take 88; the whole 166, with these copies 144).  Two copies into rows without any padding, whose products then
                // take rows in another order and put the scores back: 148.
                const char*    data   = cur.blk + (size_t)cur.h * 2 * head_data_size + (size_t)cur.bt * Cfg::kRowBytes;
                const char*    par    = cur.blk + (size_t)Hkv * 2 * head_data_size + (size_t)cur.h * 2 * head_param_sz + (size_t)cur.bt * 4;
                const int      rows   = cur.rows & 127;
                const uint32_t newest = __ballot_sync(0xffffffffu, cur.rows & 128);
                for (int l = 0; l < cnt; ++l) {
                    if (pending && (((newest >> l) & 1) || issued == STAGES)) {
                        pdl_wait();
                        pending = false;
                    }
                    ++issued;
                    if (lane == l) {
                        const uint32_t bar = full0 + 8 * s, st = stage0 + s * (uint32_t)Cfg::kStageBytes;
                        mbar_wait(empty0 + 8 * s, ph ^ 1);
                        const int n = rows * Cfg::kRowBytes, np = ((rows + 3) & ~3) * 4;
                        mbar_expect_tx(bar, 2 * (n + np));
                        constexpr int half = kTile / 2 * Cfg::kRowBytes;
                        if (rows == kTile && p.block_len == kTile) {
                            bulk_g2s_hint(st + Cfg::kOffK, data, half, bar, policy);
                            bulk_g2s_hint(st + Cfg::kOffK + Cfg::kGroupSize, data + half, 2 * half, bar, policy);
                            bulk_g2s_hint(st + Cfg::kOffV + Cfg::kGroupSize, data + 3 * half, half, bar, policy);
                            bulk_g2s_hint(st + Cfg::kOffKP, par, 2 * Cfg::kParamBytes, bar, policy);
                        }
                        else {
                            const int n0 = min(n, half);
                            bulk_g2s_hint(st + Cfg::kOffK, data, n0, bar, policy);
                            bulk_g2s_hint(st + Cfg::kOffV, data + head_data_size, n0, bar, policy);
                            if (n > n0) {
                                bulk_g2s_hint(st + Cfg::kOffK + Cfg::kGroupSize, data + half, n - n0, bar, policy);
                                bulk_g2s_hint(st + Cfg::kOffV + Cfg::kGroupSize, data + head_data_size + half, n - n0, bar, policy);
                            }
                            bulk_g2s_hint(st + Cfg::kOffKP, par, np, bar, policy);
                            bulk_g2s_hint(st + Cfg::kOffVP, par + head_param_sz, np, bar, policy);
                        }
                    }
                    __syncwarp();
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                cur = nxt;
                continue;
            }
            for (int l = 0; l < cnt; ++l) {
                const unsigned long long blk = __shfl_sync(0xffffffffu, (unsigned long long)cur.blk, l);
                const int packed = __shfl_sync(0xffffffffu, cur.h | (cur.bt << 8) | (cur.rows << 24), l);
                const int h = packed & 0xff, bt = (packed >> 8) & 0xffff, rows = (packed >> 24) & 127;
                if (pending && (((packed >> 31) & 1) || issued == STAGES)) {
                    pdl_wait();  // warp-uniform: the prologue's stores (new token's K / V, their params) are visible from here
                    pending = false;
                }
                ++issued;
                const uint32_t bar = full0 + 8 * s;
                if (lane == 0) {
                    mbar_wait(empty0 + 8 * s, ph ^ 1);
                    const int prow = (rows + 3) & ~3;
                    mbar_expect_tx(bar, 2 * rows * Cfg::kRowBytes + (Cfg::kQuant ? 2 * prow * 4 : 0));
                }
                __syncwarp();
                const uint32_t st = stage0 + s * (uint32_t)Cfg::kStageBytes;
                const char*    hb = reinterpret_cast<const char*>(blk);
                if (my_data) {
                    const int r = min(Cfg::kGroupRows, rows - my_gq * Cfg::kGroupRows);
                    if (r > 0) {
                        const char* src = hb + (size_t)(h * 2 + (my_v ? 1 : 0)) * head_data_size
                                          + (size_t)(bt + my_gq * Cfg::kGroupRows) * Cfg::kRowBytes;
                        bulk_g2s_hint(st + (my_v ? Cfg::kOffV : Cfg::kOffK) + my_gq * Cfg::kGroupSize, src,
                                      r * Cfg::kRowBytes, bar, policy);
                    }
                }
                else if (my_param) {
                    const int   prow = (rows + 3) & ~3;
                    const char* src  = hb + (size_t)Hkv * 2 * head_data_size
                                      + (size_t)(h * 2 + (my_v ? 1 : 0)) * head_param_sz + (size_t)bt * 4;
                    bulk_g2s_hint(st + (my_v ? Cfg::kOffVP : Cfg::kOffKP), src, prow * 4, bar, policy);
                }
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
            cur = nxt;
        }
        return;
    }

    // ================================== consumers ==================================
    ConsumerCtx<T, KVBITS> cx;
    cx.warp = warp;
    cx.g    = lane >> 2;
    cx.t    = lane & 3;
    const int g = cx.g, t = cx.t;
    cx.tokA  = slot_token(g, warp);
    cx.tokV0 = slot_token(2 * t, warp), cx.tokV1 = slot_token(2 * t + 1, warp);
    cx.offA  = token_smem_offset<KVBITS>(cx.tokA) + 16 * t;
    cx.offV0 = token_smem_offset<KVBITS>(cx.tokV0) + (KVBITS == 4 ? 8 : 16) * g;
    cx.offV1 = token_smem_offset<KVBITS>(cx.tokV1) + (KVBITS == 4 ? 8 : 16) * g;

    uint32_t qf[8][2];  // Q as B-operand fragments, one per k-step
    float    O[8][4];   // O^T accumulators: m-tile j -> {(slot g,head 2t),(g,2t+1),(g+8,2t),(g+8,2t+1)}
    float    M[2], L[2];
    CodeSums sums{};

    const float c = p.qk_scale;

    WorkIter it{p.batch, Hkv, p.tile_prefix};
    it.seek(lo);
    pdl_wait();  // returns at once where it has been waited for
    int       s   = 0;
    uint32_t  ph  = 0;
    long long idx = lo;

    while (idx < hi) {
        // ---------------- one segment: tiles [first_tile, first_tile + ntile) of (it.b, it.h) ----------------
        const int first_tile = it.tile;
        const int ntile      = (int)min((long long)(it.tiles - it.tile), hi - idx);
        const int k_len      = p.cu_k_len[it.b + 1] - p.cu_k_len[it.b];
        {
            if (p.fused & 1) {
                // RoPE applied in registers: every lane rotates the 4-dim chunks of its own B fragments
                const int tokq = p.cu_q_len ? p.cu_q_len[it.b] : it.b;
                const T*  qb   = reinterpret_cast<const T*>(p.q) + (size_t)tokq * p.stride + (size_t)it.h * G * kHeadDim;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint2 v = make_uint2(0u, 0u);
                    if (g < G) {
                        const int di = qk_dim0<KVBITS>(t, j);
                        T         x[4];
                        load4(qb + (size_t)g * kHeadDim + di, x);
                        if (p.q_bias) {
                            T bq[4];
                            load4(reinterpret_cast<const T*>(p.q_bias) + (size_t)(it.h * G + g) * kHeadDim + di, bq);
#pragma unroll
                            for (int i = 0; i < 4; ++i) x[i] = Ops::add(x[i], bq[i]);
                        }
                        float2 cs[2];
                        rope_cs2(cs, p.rope, p.rope_table, tokq, di, k_len - 1);
                        rope_rotate4<T>(x, cs, p.rope, di);
                        v = *reinterpret_cast<uint2*>(&x[0]);
                    }
                    qf[j][0] = v.x;
                    qf[j][1] = v.y;
                }
            }
            else {
                const T* qb = reinterpret_cast<const T*>(p.q_rot) + ((size_t)it.b * p.num_heads + (size_t)it.h * G) * kHeadDim;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint2 v = make_uint2(0u, 0u);
                    if (g < G) {
                        v = *reinterpret_cast<const uint2*>(qb + (size_t)g * kHeadDim + qk_dim0<KVBITS>(t, j));
                    }
                    qf[j][0] = v.x;
                    qf[j][1] = v.y;
                }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                O[j][0] = O[j][1] = O[j][2] = O[j][3] = 0.f;
            }
            M[0] = M[1] = -INFINITY;
            L[0] = L[1] = 0.f;
            if constexpr (kCodesInMma<T, KVBITS>) {
                sums.a[0] = sums.a[1] = sums.w[0] = sums.w[1] = 0.f;
                float q = 0.f;  // head g: this lane's 32 dims, then all 128
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float2 x = half2_to_float2(qf[j][0]), y = half2_to_float2(qf[j][1]);
                    q += (x.x + x.y) + (y.x + y.y);
                }
                q += __shfl_xor_sync(0xffffffffu, q, 1);
                q += __shfl_xor_sync(0xffffffffu, q, 2);
                sums.q[0] = __shfl_sync(0xffffffffu, q, 8 * t);
                sums.q[1] = __shfl_sync(0xffffffffu, q, 8 * t + 4);
            }
        }
        // The tile that holds the new token (position k_len - 1, always the sequence's last tile) is peeled out of the loop:
        // the out-of-line prologue call must not sit inside the loop (the ABI would pin the loop state in local memory).
        const bool peel  = (p.fused & 1) && first_tile + ntile == it.tiles;
        const int  nloop = ntile - (peel ? 1 : 0);
        // before a tile, not behind it: the peeled form takes the same steps
        auto recentre_at = [&](int tt) {
            if constexpr (kCodesInMma<T, KVBITS>) {
                if (tt > 0 && tt % kRecentre == 0) {
                    recentre<KVBITS>(O, sums);
                }
            }
        };
        int tt = 0;
        if constexpr (kTilesAtOnce<KVBITS> > 1) {
            constexpr int NT   = kTilesAtOnce<KVBITS>;
            static_assert(kRecentre % NT == 0, "the sums are centred between two turns");
            const int     many = min(nloop, it.tiles - 1 - first_tile);  // a sequence's last tile may end early
            for (; tt + NT <= many; tt += NT) {
                recentre_at(tt);
                uint32_t st[NT], done[NT];
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const bool wrap = s + i >= STAGES;
                    const int  slot = wrap ? s + i - STAGES : s + i;
                    st[i]           = stage0 + slot * (uint32_t)Cfg::kStageBytes;
                    done[i]         = empty0 + 8 * slot;
                    mbar_wait(full0 + 8 * slot, wrap ? ph ^ 1 : ph);
                }
                process_tiles<T, KVBITS, NT>(cx, st, c, qf, O, M, L, sums);
                __syncwarp();
                if (lane == 0) {
#pragma unroll
                    for (int i = 0; i < NT; ++i) mbar_arrive(done[i]);
                }
                s += NT;
                if (s >= STAGES) {
                    s -= STAGES;
                    ph ^= 1;
                }
            }
        }
        for (; tt < nloop; ++tt) {
            const int  t0      = (first_tile + tt) * kTile;
            const bool residue = t0 + kTile > k_len;
            recentre_at(tt);
            mbar_wait(full0 + 8 * s, ph);
            process_tile<T, KVBITS>(cx, stage0 + s * (uint32_t)Cfg::kStageBytes, residue, k_len, t0, c, qf, O, M, L, sums);
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(empty0 + 8 * s);
            }
            if (++s == STAGES) {
                s = 0;
                ph ^= 1;
            }
        }
        if (peel) {
            const int t0 = (it.tiles - 1) * kTile;
            recentre_at(nloop);
            mbar_wait(full0 + 8 * s, ph);
            // The new token's slot belongs to exactly one consumer warp (token_warp): that warp runs
            // the prologue for this (sequence, kv-head) -- bias, RoPE(k), quantise, store into the page for later steps -- and
            // overwrites the row the bulk copy brought in (stale bytes) in ITS OWN view of the tile; no other warp reads it.
            const int pos = k_len - 1 - t0;
            if (token_warp(pos) == warp) {
                new_token_kv<T, KVBITS>(p, it.b, it.h, k_len - 1, pos, lane, stage0 + s * (uint32_t)Cfg::kStageBytes);
                __syncwarp();
            }
            process_tile<T, KVBITS>(cx, stage0 + s * (uint32_t)Cfg::kStageBytes, true, k_len, t0, c, qf, O, M, L, sums);
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(empty0 + 8 * s);
            }
            if (++s == STAGES) {
                s = 0;
                ph ^= 1;
            }
        }
        const bool last_tile = first_tile + ntile == it.tiles;

        // ---------------- segment end: merge the 4 consumer warps, write final or partial ----------------
        if constexpr (kCodesInMma<T, KVBITS>) {
            recentre<KVBITS>(O, sums);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            L[q] += __shfl_xor_sync(0xffffffffu, L[q], 4);
            L[q] += __shfl_xor_sync(0xffffffffu, L[q], 8);
            L[q] += __shfl_xor_sync(0xffffffffu, L[q], 16);
            if constexpr (kCodesInMma<T, KVBITS>) {
                float A = sums.a[q];
                A += __shfl_xor_sync(0xffffffffu, A, 4);
                A += __shfl_xor_sync(0xffffffffu, A, 8);
                A += __shfl_xor_sync(0xffffffffu, A, 16);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float u = CodeScale<KVBITS>::unit(j);
                    O[j][q]       = fmaf(O[j][q], u, A) * (1.f / CodeScale<KVBITS>::kappa);
                    O[j][q + 2]   = fmaf(O[j][q + 2], u, A) * (1.f / CodeScale<KVBITS>::kappa);
                }
            }
        }
        if (g == 0) {
            ss.merge_M[warp][2 * t]     = M[0];
            ss.merge_M[warp][2 * t + 1] = M[1];
            ss.merge_L[warp][2 * t]     = L[0];
            ss.merge_L[warp][2 * t + 1] = L[1];
        }
        named_bar_sync(1, kConsumerWarps * 32);
        float sc[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int hd = 2 * t + q;
            float     m  = ss.merge_M[0][hd];
            for (int w = 1; w < kConsumerWarps; ++w) m = fmaxf(m, ss.merge_M[w][hd]);
            float l = 0.f;
            for (int w = 0; w < kConsumerWarps; ++w) {
                const float mw = ss.merge_M[w][hd];
                l += (mw == -INFINITY) ? 0.f : exp2_approx((mw - m) * c) * ss.merge_L[w][hd];
            }
            sc[q] = (M[q] == -INFINITY) ? 0.f : exp2_approx((M[q] - m) * c);
            if (warp == 0 && g == 0) {
                ss.final_M[hd] = m;
                ss.final_L[hd] = l;
            }
        }
        // fixed order (w0 + w2) + (w1 + w3)
        float* mo = &ss.merge_O[warp & 1][0][0];
        if (warp < 2) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int d = pv_dim<KVBITS>(g, j, 0);
                *reinterpret_cast<float2*>(mo + merge_idx(2 * t, d))     = make_float2(O[j][0] * sc[0], O[j][2] * sc[0]);
                *reinterpret_cast<float2*>(mo + merge_idx(2 * t + 1, d)) = make_float2(O[j][1] * sc[1], O[j][3] * sc[1]);
            }
        }
        named_bar_sync(1, kConsumerWarps * 32);
        if (warp >= 2) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int d  = pv_dim<KVBITS>(g, j, 0);
                float2*   a0 = reinterpret_cast<float2*>(mo + merge_idx(2 * t, d));
                float2*   a1 = reinterpret_cast<float2*>(mo + merge_idx(2 * t + 1, d));
                float2    x0 = *a0, x1 = *a1;
                x0.x += O[j][0] * sc[0], x0.y += O[j][2] * sc[0];
                x1.x += O[j][1] * sc[1], x1.y += O[j][3] * sc[1];
                *a0 = x0, *a1 = x1;
            }
        }
        named_bar_sync(1, kConsumerWarps * 32);
        const bool complete = (first_tile == 0) && last_tile;
        const int  ctid     = threadIdx.x;  // 0..127
        const float* m0     = &ss.merge_O[0][0][0];
        const float* m1     = &ss.merge_O[1][0][0];
        if (complete) {
            for (int i = ctid; i < G * kHeadDim / 2; i += kConsumerWarps * 32) {
                const int    hd  = (2 * i) / kHeadDim;
                const int    d   = (2 * i) % kHeadDim;
                const float  inv = 1.f / ss.final_L[hd];
                const int    mi  = merge_idx(hd, d);
                const float2 a = *reinterpret_cast<const float2*>(m0 + mi), b2 = *reinterpret_cast<const float2*>(m1 + mi);
                const int    col = it.h * G * kHeadDim + 2 * i;
                T*           dst = reinterpret_cast<T*>(p.out)
                         + (p.out_mt > 0 ? ((size_t)(col >> 3) * p.out_mt + it.b) * 8 + (col & 7) :
                                           (size_t)it.b * p.out_stride + col);
                *reinterpret_cast<uint32_t*>(dst) = Ops::pack2((a.x + b2.x) * inv, (a.y + b2.y) * inv);
            }
        }
        else {
            const int slot = 2 * blockIdx.x + (idx == lo ? 0 : 1);
            float*    po   = p.partial_O + (size_t)slot * kMaxGroup * kHeadDim;
            for (int i = ctid; i < G * kHeadDim / 2; i += kConsumerWarps * 32) {
                const int    hd = (2 * i) / kHeadDim, d = (2 * i) % kHeadDim;
                const int    mi = merge_idx(hd, d);
                const float2 a = *reinterpret_cast<const float2*>(m0 + mi), b2 = *reinterpret_cast<const float2*>(m1 + mi);
                *reinterpret_cast<float2*>(po + 2 * i) = make_float2(a.x + b2.x, a.y + b2.y);
            }
            if (ctid < G) {
                p.partial_ML[((size_t)slot * kMaxGroup + ctid) * 2]     = ss.final_M[ctid];
                p.partial_ML[((size_t)slot * kMaxGroup + ctid) * 2 + 1] = ss.final_L[ctid];
            }
            if (p.fused & 2) {
                // In-kernel fix-up: arrive on the segment's counter (the CTA barrier orders every thread's partial stores
                // before thread 0's gpu-scope acq_rel atomic); the CTA that arrives LAST merges all partials of the segment
                // in CTA order -- the same sum whoever merges -- and re-arms the counter.
                named_bar_sync(1, kConsumerWarps * 32);
                if (ctid == 0) {
                    ss.seg        = segment_ctas(p, it.b, it.h, p.grid_main);
                    int*      ctr = p.seg_counters + ss.seg.cf;  // one segment at most leaves a CTA at its range's end
                    const int old = atom_add_acq_rel_gpu(ctr, 1);
                    ss.fix_last   = (old == ss.seg.n - 1);
                    if (old == ss.seg.n - 1) {
                        *ctr = 0;  // every piece of the segment has arrived: nobody touches the counter again in this launch
                    }
                }
                named_bar_sync(1, kConsumerWarps * 32);
                if (ss.fix_last) {
                    merge_segment<T>(p, it.b, it.h, ss.seg, p.grid_main, ctid, kConsumerWarps * 32);
                }
            }
        }
        named_bar_sync(1, kConsumerWarps * 32);

        // advance to the next segment
        idx += ntile;
        it.tile += ntile - 1;
        it.next();
    }
}

// Fix-up reduction as a separate kernel (used when the in-kernel fix-up is off).
template<class T>
__global__ void __launch_bounds__(256) decode_reduce_kernel(const __grid_constant__ KernelParams p, int grid_main)
{
    pdl_launch_dependents();
    pdl_wait();
    const int b     = blockIdx.y;
    const int h     = blockIdx.x;
    const int tiles = p.tile_prefix[b + 1] - p.tile_prefix[b];
    if (tiles == 0) {
        return;
    }
    __shared__ SegCtas s_seg;
    if (threadIdx.x == 0) {
        s_seg = segment_ctas(p, b, h, grid_main);
    }
    __syncthreads();
    if (s_seg.n <= 1) {
        return;  // written directly by the main kernel
    }
    merge_segment<T>(p, b, h, s_seg, grid_main, threadIdx.x, blockDim.x);
}

// decode_merge.cu: the fix-up of few segments with many pieces each, when it is the better one and its launch
bool few_segments(const KernelParams& p, int grid_main);
int  launch_reduce_heads(bool bf16, const KernelParams& p, int grid_main, cudaStream_t st);

}  // namespace attn
}  // namespace b200
