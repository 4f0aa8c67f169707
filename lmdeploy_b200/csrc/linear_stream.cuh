// Dense linear layer with many output features and more than 64 tokens (a vocabulary head): a persistent tcgen05 kernel, one CTA per SM.
//
// Y[tokens, N] = X . W with the prepared weights and packed activations of gemm.cuh.  What differs:
//   * tokens are the M side of the product (at more than 64 they fill it) and features the N side, so an accumulator row is a token
//     and the epilogue stores 16 bytes of consecutive features per thread;
//   * two tiles of 128 features share every activation tile: at 128 tokens a tile of X is as large as a tile of weights, and with
//     one tile per CTA half of what an SM takes in is X;
//   * a CTA owns a contiguous range of tiles and its ring never drains between them: the accumulators of a pair alternate between
//     two halves of tensor memory, so the epilogue warps store one pair while the next one is multiplied;
//   * a stage is half a k-group (64 k's: 16 KB of weights per tile, MT * 128 bytes of X), its copies issued by one lane each.
//     (Pieces of 2 KB, which would let one multiplication take all 256 features, are issue-bound: 203 us for 176 below.)
// Measured, 128 tokens, f16 4096 x 128256: 195 -> 176 us in a short run; in a long one the card's power limit (990 W, SM clock down
// to 0.9 GHz) bounds it, 231 -> 213.  First calls on freshly prepared weights, both kernels in one process: after a second of idling 202 -> 182; behind
// 1.5 s of repeated calls of this kernel 285 -> 235, of gemm_kernel 238 -> 198 (the card is still at the lower clocks; the preparation, unchanged,
// takes 3.7, 5.3 and 4.5 ms there).  Pairs of tiles dealt out in turn, so that all CTAs walk one window, made no difference to either.
#pragma once

#include "gemm.cuh"

namespace b200 {
namespace gemm {

constexpr int kStreamStages  = 4;
constexpr int kStreamWBytes  = kDenseBlockBytes / 2;
constexpr int kStreamThreads = 32 * 10;  // producer, MMA issuer, eight epilogue warps (tile, quarter of the rows)

constexpr int stream_stage_bytes(int MT)
{
    return 2 * kStreamWBytes + MT * 128;
}
// the 128 - MT rows that the multiplication reads past a stage's X (their results are not used) end within the allocation
constexpr int stream_smem_bytes(int MT)
{
    return kStreamStages * stream_stage_bytes(MT) + (128 - MT) * 16;
}

template<class T>
__global__ void __launch_bounds__(kStreamThreads, 1) linear_stream_kernel(const Params p)
{
    using Ops = TypeOps<T>;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar_full[kStreamStages], bar_empty[kStreamStages], bar_dfull[2], bar_dempty[2];
    __shared__ uint32_t s_tmem;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int tiles = p.N / kBN, lo = (int)((int64_t)tiles * blockIdx.x / gridDim.x), hi = (int)((int64_t)tiles * (blockIdx.x + 1) / gridDim.x);
    const int steps = p.K / kKG * 2;  // stages per pair of tiles
    const int XB = p.MT * 128, SB = stream_stage_bytes(p.MT);
    pdl_launch_dependents();
    if (threadIdx.x < kStreamStages) {
        mbar_init(smem_u32(&bar_full[threadIdx.x]), 1);
        mbar_init(smem_u32(&bar_empty[threadIdx.x]), 1);
        fence_mbar_init();
    }
    else if (threadIdx.x < kStreamStages + 2) {
        mbar_init(smem_u32(&bar_dfull[threadIdx.x - kStreamStages]), 1);
        mbar_init(smem_u32(&bar_dempty[threadIdx.x - kStreamStages]), 8);
        fence_mbar_init();
    }
    if (warp == 1) {
        umma::tmem_alloc(smem_u32(&s_tmem), 512);
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s_tmem, ring = smem_u32(smem);

    if (warp == 0) {
        // ================================ producer ================================
        const uint64_t pol = make_evict_first_policy();
        struct Pos {
            int tile, step;
        };
        auto next = [&](Pos& q) {
            if (++q.step == steps) {
                q.step = 0, q.tile += 2;
            }
        };
        auto arm = [&](const Pos& q, int s) {
            if (lane == 0) {
                mbar_expect_tx(smem_u32(&bar_full[s]), min(2, hi - q.tile) * kStreamWBytes + XB);
            }
            __syncwarp();
        };
        auto fetch_w = [&](const Pos& q, int s) {
            if (lane < min(2, hi - q.tile)) {
                bulk_g2s_hint(ring + s * SB + lane * kStreamWBytes, p.w + ((size_t)(q.tile + lane) * steps + q.step) * kStreamWBytes, kStreamWBytes, smem_u32(&bar_full[s]), pol);
            }
        };
        auto fetch_x = [&](const Pos& q, int s) {
            if (lane == 2) {
                bulk_g2s(ring + s * SB + 2 * kStreamWBytes, reinterpret_cast<const uint8_t*>(p.xp) + (size_t)q.step * XB, XB, smem_u32(&bar_full[s]));
            }
        };
        Pos w{lo, 0}, x{lo, 0};
        for (int s = 0; s < kStreamStages && w.tile < hi; ++s, next(w)) {  // weights are constants: ahead of the previous kernel's end
            arm(w, s);
            fetch_w(w, s);
        }
        pdl_wait();
        for (int s = 0; s < kStreamStages && x.tile < hi; ++s, next(x)) {
            fetch_x(x, s);
        }
        int      s  = 0;
        uint32_t ph = 0;
        for (; w.tile < hi; next(w)) {
            if (lane == 0) {
                mbar_wait(smem_u32(&bar_empty[s]), ph);
            }
            __syncwarp();
            arm(w, s);
            fetch_w(w, s);
            fetch_x(w, s);
            if (++s == kStreamStages) {
                s = 0, ph ^= 1;
            }
        }
    }
    else if (warp == 1) {
        // ================================ MMA issuer ================================
        constexpr bool bf     = std::is_same<T, nv_bfloat16>::value;
        const uint32_t a_step = (uint32_t)(2 * p.MT * 16) >> 4, b_step = (uint32_t)(2 * kBN * 16) >> 4;
        const uint32_t idesc  = umma::make_idesc_f16(128, kBN, bf);
        int            s = 0, b = 0;
        uint32_t       ph = 0, phd = 1;
        for (int tile = lo; tile < hi; tile += 2) {
            const int n = min(2, hi - tile);
            mbar_wait(smem_u32(&bar_dempty[b]), phd);
            umma::fence_after_sync();
            for (int i = 0; i < steps; ++i) {
                mbar_wait(smem_u32(&bar_full[s]), ph);
                umma::fence_after_sync();
                const uint64_t ad = umma::make_smem_desc(ring + s * SB + 2 * kStreamWBytes, p.MT * 16, 128);
                const uint64_t bd = umma::make_smem_desc(ring + s * SB, kBN * 16, 128);
                if (elect_one()) {
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (t < n) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                umma::mma_f16_ss(tmem + b * 256 + t * kBN, ad + (uint64_t)(ks * a_step), bd + (uint64_t)(t * (kStreamWBytes >> 4) + ks * b_step), idesc, i > 0 || ks > 0);
                            }
                        }
                    }
                    umma::commit(smem_u32(&bar_empty[s]));
                    if (i == steps - 1) {
                        umma::commit(smem_u32(&bar_dfull[b]));
                    }
                }
                __syncwarp();
                if (++s == kStreamStages) {
                    s = 0, ph ^= 1;
                }
            }
            if ((b ^= 1) == 0) {
                phd ^= 1;
            }
        }
    }
    else {
        // ================================ epilogue: thread = token, warp = (32 tokens, tile) ================================
        const int      t = (warp - 2) >> 2, q = warp & 3, tok = 32 * q + lane;
        const uint32_t row   = tmem + ((uint32_t)(32 * q) << 16) + t * kBN;
        const bool     gated = p.epilogue == 1;
        T*             y     = reinterpret_cast<T*>(p.y);
        const T*       bias  = reinterpret_cast<const T*>(p.bias);
        int            b     = 0;
        uint32_t       ph    = 0;
        pdl_wait();  // an earlier kernel may still read the output's memory
        for (int tile = lo; tile < hi; tile += 2) {
            mbar_wait(smem_u32(&bar_dfull[b]), ph);
            umma::fence_after_sync();
            if (tile + t < hi && 32 * q < p.M) {
                const int n0 = (tile + t) * kBN;
                for (int c = 0; c < kBN; c += 16) {
                    uint32_t v[16];
                    umma::ld_32x32b_x16(row + b * 256 + c, v);
                    umma::wait_ld();
                    float f[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]) + (bias ? Ops::to_f32(bias[n0 + c + i]) : 0.f);
                    if (tok < p.M) {
                        if (gated) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) f[i] = __fdividef(f[2 * i], 1.f + __expf(-f[2 * i])) * f[2 * i + 1];
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (h == 0 || !gated) {
                                const int   n = (gated ? (n0 + c) / 2 : n0 + c) + h * 8;
                                const uint4 o = make_uint4(Ops::pack2(f[h * 8], f[h * 8 + 1]), Ops::pack2(f[h * 8 + 2], f[h * 8 + 3]), Ops::pack2(f[h * 8 + 4], f[h * 8 + 5]),
                                                           Ops::pack2(f[h * 8 + 6], f[h * 8 + 7]));
                                *reinterpret_cast<uint4*>(p.out_mode == 0 ? y + (size_t)tok * p.ldy + n : y + ((size_t)(n >> 3) * p.out_mt + tok) * 8) = o;
                            }
                        }
                    }
                }
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_u32(&bar_dempty[b]));
            }
            if ((b ^= 1) == 0) {
                ph ^= 1;
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        umma::tmem_dealloc(tmem, 512);
    }
}

}  // namespace gemm
}  // namespace b200
