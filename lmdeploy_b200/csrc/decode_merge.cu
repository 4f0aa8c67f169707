// Fix-up of decode attention for few segments (decode_attention.cuh: decode_reduce_kernel takes the rest).
#include "decode_attention.cuh"
#include "host_utils.h"

namespace b200 {
namespace attn {

// Few segments have many pieces each (four or more on average): merge_segment's threads would read eight of them at a
// time, each batch behind the one before, on one SM per segment.  Here a CTA takes one query head; its warps copy the pieces of it into
// shared memory, up to 64 at once, and a thread sums one dimension in the same order with the same roundings, so no output depends on
// which of the two kernels ran.
// us, whole operator, captured calls, decode_reduce_kernel -> this: three sequences of 37 - 7001 bf16 tokens, 48 / 8 heads, 26.4 -> 19.7; one of 4096
// int8 tokens, 32 / 8 heads, 32.6 -> 12.6; one of 8000 int4 tokens, 8 / 2 heads, 63 -> 16.2; at the line twelve of 700 - 1500 int8 tokens, 32 / 8 heads,
// 19.0 -> 16.4, and 37 of 5000 - 5496, 8 / 2 heads, 31.0 -> 27.2.  (All loads of a thread in registers instead, 32 or 64 at once: 21.0 for 19.7.)
constexpr int kReduceBatch = 64;

B200_DEVICE int merge_slot(const SegCtas& sg, int grid_main, int k)  // as merge_segment has it
{
    if (sg.sparse) {
        return 2 * (int)(((sg.s0 + k + 1) * grid_main - 1) / sg.total);  // one unit per CTA: always its first slot
    }
    return 2 * (sg.cf + k) + (k == 0 ? sg.first_slot : 0);
}

bool few_segments(const KernelParams& p, int grid_main)
{
    return grid_main >= 4 * p.num_kv_heads * p.batch;
}

template<class T>
__global__ void __launch_bounds__(kHeadDim) decode_reduce_heads_kernel(const __grid_constant__ KernelParams p, int grid_main)
{
    using Ops = TypeOps<T>;
    __shared__ __align__(16) float s_o[kReduceBatch][kHeadDim];
    __shared__ int    s_slot[kReduceBatch];  // where the pieces lie
    __shared__ float2 s_wl[kReduceBatch];    // their weight and sum
    __shared__ float  s_top[kHeadDim / 32];
    pdl_launch_dependents();
    pdl_wait();
    const int G = p.num_heads / p.num_kv_heads, b = blockIdx.y, h = blockIdx.x / G, hd = blockIdx.x - h * G, d = threadIdx.x;
    if (p.tile_prefix[b + 1] == p.tile_prefix[b]) {
        return;
    }
    const SegCtas sg = segment_ctas(p, b, h, grid_main);
    if (sg.n <= 1) {
        return;  // written directly by the main kernel
    }
    auto read = [&](int slot) { return __ldcg(reinterpret_cast<const float2*>(&p.partial_ML[((size_t)slot * kMaxGroup + hd) * 2])); };
    // pieces k1 .. k1 + kReduceBatch - 1: their slots, and copies of their values on the way
    auto fetch = [&](int k1) {
        const int n = min(sg.n - k1, kReduceBatch);
        if (d < n) {
            s_slot[d] = merge_slot(sg, grid_main, k1 + d);
        }
        __syncthreads();
        for (int k = d >> 5; k < n; k += kHeadDim / 32) {
            const int i = (d & 31) * 4;
            cp_async16(smem_u32(&s_o[k][i]), &p.partial_O[((size_t)s_slot[k] * kMaxGroup + hd) * kHeadDim + i]);
        }
        return n;
    };
    int    n  = fetch(0);
    float2 ml = d < n ? read(s_slot[d]) : make_float2(-INFINITY, 0.f);
    float  m  = ml.x;
    for (int k = kReduceBatch + d; k < sg.n; k += kHeadDim) m = fmaxf(m, read(merge_slot(sg, grid_main, k)).x);
#pragma unroll
    for (int x = 16; x >= 1; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
    if ((d & 31) == 0) {
        s_top[d >> 5] = m;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kHeadDim / 32; ++w) m = fmaxf(m, s_top[w]);
    float acc = 0.f, l = 0.f;
    for (int k1 = 0;;) {
        if (d < n) {
            s_wl[d] = make_float2(ml.x == -INFINITY ? 0.f : exp2_approx((ml.x - m) * p.qk_scale), ml.y);
        }
        cp_async_wait_all();
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const float2 wl = s_wl[k];
            l += wl.x * wl.y;
            acc += wl.x * s_o[k][d];
        }
        if ((k1 += kReduceBatch) >= sg.n) {
            break;
        }
        __syncthreads();  // read by everyone
        n = fetch(k1);
        if (d < n) {
            ml = read(s_slot[d]);
        }
    }
    const int col = blockIdx.x * kHeadDim + d;
    T*        out = reinterpret_cast<T*>(p.out);
    out[p.out_mt > 0 ? ((size_t)(col >> 3) * p.out_mt + b) * 8 + (col & 7) : (size_t)b * p.out_stride + col] = Ops::from_f32(acc / l);
}

int launch_reduce_heads(bool bf16, const KernelParams& p, int grid_main, cudaStream_t st)
{
    launch_k(bf16 ? decode_reduce_heads_kernel<nv_bfloat16> : decode_reduce_heads_kernel<half>, dim3(p.num_heads, p.batch), dim3(kHeadDim), 0, st, p, grid_main);
    return check_launch("decode_reduce_heads_kernel");
}

}  // namespace attn
}  // namespace b200
