// Weight-only-quant linear layer for a few tokens (m <= 24) on mma.sync.
//
// The tcgen05 kernel (gemm.cuh) owns 128 or 256 output features per CTA, so a projection has to cut K over several CTAs to use the
// chip and pay for the exchange of their partial sums, wants the activations in a packed layout (a launch of its own), and fills
// at least 16 token columns whatever m is.  With few tokens none of that buys anything: the work is the weight stream.  Here
//   * a CTA owns R = 16..128 output features over ALL of K, so nothing is exchanged between CTAs.  Its eight warps are 8 / kw row
//     groups of 16 * RT features times kw warps along K (every kw-th group of 128 k's); the sums of the kw warps meet in shared
//     memory at the end, in warp order (deterministic);
//   * weights go from global memory into registers, DEPTH k-groups ahead: a lane (g = lane / 4, t = lane % 4) reads 32 contiguous
//     bytes of the prepared stream = the 16-byte units of features 2g and 2g + 1 for one set of k's, the two rows of an m16n8k16 A
//     fragment that it holds.  Which k's the columns of a fragment stand for is free as long as the B fragment (8 tokens of X)
//     uses the same ones, so nothing is shuffled;
//   * X is read in place (row-major) by bulk copies into a ring of shared memory, kw k-groups of every token per stage, and from
//     there by the lane that needs it.
// u4 weights become the same T(fma(q, s, t)) as in the tcgen05 kernel, e4m3 weights the same T(weight * scale).
//
// Measured (us, captured b200_linear_forward, pack and tcgen05 kernel -> this kernel): u4 f16 m 1 4096 x 6144 11.4 -> 7.1, 4096 x 4096
// 10.0 -> 4.7, 14336 x 4096 14.3 -> 10.9, 1024 x 1536 6.3 -> 2.1; fp8 m 8 8192 x 10240 31.9 -> 25.0; dense m 1 14336 x 4096 24.8 -> 19.9.
// Small layers are bound by the latency of one launch, large u4 layers by the integer pipe (the unpacking, 57 % busy on the
// fullest SM) and by how few warps 128 registers leave (4 a scheduler): the tcgen05 kernel takes those.  Weights by bulk copies into
// shared memory instead (rows of 16..64 features are pieces of 256 to 1024 bytes) took twice as long; bulk prefetches into L2 ahead
// of the loads changed 6.3 to 6.2 and 15.6 to 17.5.
#pragma once

#include "gemm.cuh"

namespace b200 {
namespace gemm {

constexpr int kThinWarps     = 8;
constexpr int kThinThreads   = 32 * kThinWarps;
constexpr int kThinMaxStages = 4;
constexpr int kThinSmem      = 104 * 1024;              // two CTAs per SM

struct ThinParams {
    int64_t x_tok;   // bytes between tokens of X
    int     kw;      // warps that share a CTA's rows and take every kw-th k-group: 1, 2, 4 or 8
    int     stages;  // X ring: a stage holds kw k-groups of every token
    int     pitch;   // bytes between tokens of a stage
};

// 32 bytes of weights: read once, so not kept in L1
B200_DEVICE void ldg256(uint32_t (&v)[8], const void* p)
{
    asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "l"(p));
}

template<class T, int FMT, int RT, int NT, int DEPTH>
__global__ void __launch_bounds__(kThinThreads, 2) linear_thin_kernel(const Params p, const ThinParams tp)
{
    using Ops            = TypeOps<T>;
    constexpr int  LW    = FMT == kU4 ? 1 : FMT == kDense ? 4 : 2;  // 32-byte loads per (16 rows, k-group) and lane
    constexpr int  WB    = block_bytes_of(FMT);
    static_assert(WB % 32 == 0, "a lane's 32 bytes of any block are aligned");
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar_full[kThinMaxStages], bar_empty[kThinMaxStages];

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int kgs = p.K / kKG, KW = tp.kw, steps = (kgs + KW - 1) / KW;
    const int R   = 16 * RT * kThinWarps / KW;  // output features of this CTA
    const int n0  = blockIdx.x * R;
    const int xs  = NT * 8 * tp.pitch;          // bytes of an X stage
    pdl_launch_dependents();
    if (threadIdx.x < 2 * kThinMaxStages) {
        const int i = threadIdx.x;
        mbar_init(smem_u32(i < kThinMaxStages ? &bar_full[i] : &bar_empty[i - kThinMaxStages]), i < kThinMaxStages ? 1 : kThinWarps);
        fence_mbar_init();
    }
    __syncthreads();

    // stage j % stages <- the KW groups of step j of every token's row: a lane per token
    auto fetch_x = [&](int j) {
        const int      u     = j % tp.stages, fill = j / tp.stages;
        const uint32_t bytes = min(KW, kgs - j * KW) * (kKG * 2), bar = smem_u32(&bar_full[u]);
        if (lane == 0) {
            if (fill > 0) {
                mbar_wait(smem_u32(&bar_empty[u]), (fill - 1) & 1);
            }
            mbar_expect_tx(bar, bytes * p.M);
        }
        __syncwarp();
        if (lane < p.M) {
            bulk_g2s(smem_u32(smem) + u * xs + lane * tp.pitch, reinterpret_cast<const uint8_t*>(p.xp) + lane * tp.x_tok + (size_t)j * KW * (kKG * 2), bytes, bar);
        }
    };

    const int rw = warp / KW, kw = warp - rw * KW;
    // weights: block (n0 / 128, kg); within it this lane's 32 bytes of load l, row tile r
    const uint8_t* wblk = p.w + (size_t)(n0 / kBN) * kgs * WB;
    const int      row0 = n0 % kBN + rw * (16 * RT) + 2 * g;
    uint32_t       w[DEPTH][RT][LW][8];
    uint2          par[DEPTH][RT];  // u4: (s, t) of the two rows; fp8: their scales
    auto           load_w = [&](int st, int kg) {
        const uint8_t* b = wblk + (size_t)kg * WB;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
#pragma unroll
            for (int l = 0; l < LW; ++l) {
                ldg256(w[st][r][l], b + ((l * 4 + t) * kBN + row0 + r * 16) * 16);
            }
            if constexpr (FMT == kU4 || FMT == kFp8Col) {
                par[st][r] = __ldg(reinterpret_cast<const uint2*>(b + (FMT == kU4 ? 8192 : 16384) + (row0 + r * 16) * 4));
            }
        }
    };
    // from here on: weights (the kernel ahead may be the one that writes them: no pack stands between), activations, an output that
    // an earlier kernel may still read
    pdl_wait();
#pragma unroll
    for (int s = 0; s < DEPTH; ++s) {
        if (kw + s * KW < kgs) {
            load_w(s, kw + s * KW);
        }
    }
    bool dn = false;
    if constexpr (FMT == kU4 && std::is_same<T, half>::value) {
        dn = __ldg(p.u4_fast) != 0;
    }
    if (warp == 0) {
        for (int j = 0; j < min(tp.stages, steps); ++j) {
            fetch_x(j);
        }
    }

    float acc[RT][NT][4];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][j][c] = 0.f;

    // the 16-byte chunk of 8 k's that unit `i` (0..3) of this lane's k's in the group stands for
    auto chunk   = [&](int i) { return FMT == kU4 ? t * 4 + i : FMT == kDense ? i * 4 + t : ((i >> 1) * 4 + t) * 2 + (i & 1); };
    auto compute = [&](auto DN, int st, uint32_t xsm) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // 8 k's of each of the two rows
            uint4 x[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) x[j] = lds128(xsm + j * 8 * tp.pitch + chunk(i) * 16);
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                uint32_t a0[4], a1[4];     // k pairs (0,1) (2,3) (4,5) (6,7) of rows 2g and 2g + 1
                if constexpr (FMT == kU4) {
                    auto unpack = [&](uint32_t q, uint32_t pr, uint32_t(&o)[4]) {
                        const uint32_t s2 = __byte_perm(pr, pr, 0x1010), t2 = __byte_perm(pr, pr, 0x3232);
                        uint32_t       h[4];
                        if constexpr (decltype(DN)::value) {
                            h[0] = (q << 4) & kU4FastMask;
                            h[1] = q & kU4FastMask;
                            h[2] = (q >> 4) & kU4FastMask;
                            h[3] = __funnelshift_r(q, q, 8) & kU4FastMask;
                        }
                        else {
                            Ops::cvt_u4x8(q, h);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) o[e] = Ops::fma2(h[e], s2, t2);
                    };
                    unpack(w[st][r][0][i], par[st][r].x, a0);
                    unpack(w[st][r][0][4 + i], par[st][r].y, a1);
                }
                else if constexpr (FMT == kDense) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) a0[e] = w[st][r][i][e], a1[e] = w[st][r][i][4 + e];
                }
                else {
                    const uint32_t s0 = __byte_perm(par[st][r].x, 0, 0x1010), s1 = __byte_perm(par[st][r].y, 0, 0x1010);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint32_t q0 = w[st][r][i >> 1][(i & 1) * 2 + (e >> 1)], q1 = w[st][r][i >> 1][4 + (i & 1) * 2 + (e >> 1)];
                        a0[e] = Ops::mul2(e4m3x2_to<T>(e & 1 ? q0 >> 16 : q0 & 0xffffu), s0);
                        a1[e] = Ops::mul2(e4m3x2_to<T>(e & 1 ? q1 >> 16 : q1 & 0xffffu), s1);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t a[4] = {a0[2 * h], a1[2 * h], a0[2 * h + 1], a1[2 * h + 1]};
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const uint32_t b[2] = {h ? x[j].z : x[j].x, h ? x[j].w : x[j].y};
                        Ops::mma16816(acc[r][j], a, b);
                    }
                }
            }
        }
    };
    auto loop = [&](auto DN) {
        int       xstage = 0;
        uint32_t  ph     = 0;
        const int lag    = tp.stages > 2 ? 2 : 1;
        for (int i0 = 0; i0 < steps; i0 += DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; ++d) {
                const int i = i0 + d, kg = i * KW + kw;
                if (i < steps) {
                    // refill the stage of `lag` steps ago, the warps in turn
                    const int j = i - lag + tp.stages;
                    if (i >= lag && j < steps && warp == i % kThinWarps) {
                        fetch_x(j);
                    }
                    mbar_wait(smem_u32(&bar_full[xstage]), ph);
                    if (kg < kgs) {
                        compute(DN, d, smem_u32(smem) + xstage * xs + g * tp.pitch + kw * (kKG * 2));
                        if (kg + DEPTH * KW < kgs) {
                            load_w(d, kg + DEPTH * KW);
                        }
                    }
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(smem_u32(&bar_empty[xstage]));
                    }
                    if (++xstage == tp.stages) {
                        xstage = 0, ph ^= 1;
                    }
                }
            }
        }
    };
    if (dn) {
        loop(std::true_type{});
    }
    else {
        loop(std::false_type{});
    }

    // sums of the KW warps that share rows: [kw][token][row], pitch R + 4 words (a warp's float2 stores hit distinct banks); the X
    // stages are idle by now
    float* red = reinterpret_cast<float*>(smem);
    __syncthreads();
    const int rp = R + 4;
#pragma unroll
    for (int r = 0; r < RT; ++r) {
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            float* d = red + (size_t)(kw * NT * 8 + j * 8 + 2 * t) * rp + rw * (16 * RT) + r * 16 + 2 * g;
            *reinterpret_cast<float2*>(d)      = make_float2(acc[r][j][0], acc[r][j][2]);
            *reinterpret_cast<float2*>(d + rp) = make_float2(acc[r][j][1], acc[r][j][3]);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < p.M * (R / 2); i += 32 * kThinWarps) {
        const int tok = i / (R / 2), c = i % (R / 2) * 2;
        float2    s = make_float2(0.f, 0.f);
        for (int k = 0; k < KW; ++k) {
            const float2 v = *reinterpret_cast<const float2*>(red + (size_t)(k * NT * 8 + tok) * rp + c);
            s.x += v.x, s.y += v.y;
        }
        finalize_pair<T>(p, tok, n0 + c, s.x, s.y);
    }
}

}  // namespace gemm
}  // namespace b200
