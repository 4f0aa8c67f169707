// Windowed, chunked or causal softmax attention of hybrid decoders on tcgen05 tensor cores, in one pass over the keys: for the heads
// that are scored one by one (no recombination across heads, no cap, no distance penalty), bf16 pages, 64 or 128 dimensions.
// b200h_window_attention chooses it (flash_attention_fits, flash_attention_pays); the two-pass kernels of window_attention.cuh remain for the rest.
// Included by hybrid_ops.cu inside namespace b200h, after window_attention.cuh.
//
// Precision: keys and values are bf16 in the cache, so they enter the products as they are; a float query is taken as the sum of two bf16
// parts, which keeps 17 of its 24 bits, a softmax weight likewise, and each product is the sum of two tensor-core products with float
// accumulators.  That is less than the two-pass kernels hold and far more than the bf16 result shows: over seven steps of 180 - 4096 rows
// (three kinds of attention, up to 2048 keys behind) the error against 64 bits is the same to four digits (2.44e-3 - 5.09e-3).
// Rescaling an accumulator only when a maximum has grown a lot is the published technique of FlashAttention's later versions.
//
// A UNIT is up to UNIT_ROWS consecutive rows of one sequence, a PIECE a unit and a key/value head.  A piece makes two UMMA tiles of
// 128 rows (row = token * rep + head in group): one map per head: two blocks of 128 / rep tokens; two maps: the same tokens' first and
// second maps, which share the values.  Roles of a block (one per SM, persistent over pieces dealt out largest first):
//   warps 0-3 / 4-7   softmax of tile 0 / 1, thread = row; accumulator in tensor memory, rescaled when a row's maximum grew by > 2^8;
//                     sink, head norm, gate and the subtraction of the maps at the end, straight to T
//   warp 8            issues the tensor-core products
//   warps 9-15        keys and values of 128 positions at a time, by 16-byte asynchronous copies from the pages
// Measured (B200, 4 x 1024 rows of causal attention, 16 / 8 heads of 128, with the projection): 2034 us by the two passes, which
// multiply on the float units, 154 us here (projection 53, preparation 22, plan 9, this kernel 79 us).  What bounds it: 16-byte copies enter shared memory at one per cycle and
// SM (2 k cycles for 32 KB whatever their pattern), and a piece's start.

using b200::smem_u32;

constexpr int kFaKeys = 128, kFaThreads = 512, kFaLoaders = 7;
constexpr int kFaLazy = 8;              // log2 of the growth of a row's maximum that forces a rescale of the accumulator

struct FlashArgs {
    int n, heads, kv_heads, block_len, window, keep, chunk;
    int gate_div, out_norm;
    float scale, lambda, out_scale, eps;
    const float* qn;                    // [n, heads * maps * D]
    const bf16* gate;                   // nullptr: none
    int64_t ld_gate;
    const float* sink;                  // [heads * maps] or nullptr
    const int* tok_seq;
    const int* tok_pos;
    const int64_t* block_ptrs;
    const int* cu_blocks;
    int64_t layer_off, v_off;
    bf16* y;
    int64_t ld_y;
    float* second;                      // maps 2: scratch [n, heads * vdim] for the second map's outputs
    int* plan;                          // [4 + n + 8 n] ints: unit count, -, first rows of units, units in order of work
};

struct FlashUnit { int row, count, pos, seq, first, kept, tiles, pad; };      // first: first key tile of the window; kept: tiles in front of it

__device__ __forceinline__ FlashUnit* flash_units(const FlashArgs& a) { return reinterpret_cast<FlashUnit*>(a.plan + (4 + a.n + 3) / 4 * 4); }

__device__ __forceinline__ int flash_lo(const FlashArgs& a, int pos)         // first key of the row's window or chunk
{
    const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    return a.chunk > 0 ? max(lo, pos / a.chunk * a.chunk) : lo;
}

// One block: rows -> units (runs of one sequence, cut every `rows`), sorted by their number of key tiles, largest first.
__global__ void __launch_bounds__(1024) flash_plan_kernel(const FlashArgs a, int rows)
{
    __shared__ int warps[32], bins[1024], total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, per = (a.n + 1023) / 1024, t0 = min(a.n, tid * per), t1 = min(a.n, t0 + per);
    auto starts_run = [&](int t) { return t == 0 || a.tok_seq[t] != a.tok_seq[t - 1] || a.tok_pos[t] != a.tok_pos[t - 1] + 1; };
    // inclusive scans over the block: of a sum, and of the largest value
    auto scan = [&](int v, bool sum) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v = sum ? v + u : max(v, u);
        }
        __syncthreads();                    // warps[] may still be read from an earlier scan
        if (lane == 31) warps[warp] = v;
        __syncthreads();
        int w = lane < warp ? warps[lane] : (sum ? 0 : -1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int u = __shfl_xor_sync(0xffffffffu, w, o);
            w = sum ? w + u : max(w, u);
        }
        return sum ? v + w : max(v, w);
    };
    int* first = a.plan + 4;
    // the run that a thread's first row belongs to: the latest run start before it
    int run = -1;
    for (int t = t0; t < t1; ++t) if (starts_run(t)) run = t;
    bins[tid] = scan(run, false);
    __syncthreads();
    const int before = tid > 0 ? bins[tid - 1] : -1;
    int count = 0;
    run = before;
    for (int t = t0; t < t1; ++t) {
        if (starts_run(t)) run = t;
        count += (t - run) % rows == 0;
    }
    __syncthreads();
    int at = scan(count, true);
    if (tid == 1023) total = at;
    bins[tid] = 0;
    at -= count;
    run = before;
    for (int t = t0; t < t1; ++t) {
        if (starts_run(t)) run = t;
        if ((t - run) % rows == 0) first[at++] = t;
    }
    __syncthreads();
    const int units = total;
    auto unit_of = [&](int u) {
        FlashUnit x;
        x.row = first[u];
        x.count = (u + 1 < units ? first[u + 1] : a.n) - x.row;
        x.pos = a.tok_pos[x.row];
        x.seq = a.tok_seq[x.row];
        x.first = flash_lo(a, x.pos) / kFaKeys;
        x.kept = (min(a.keep, x.first * kFaKeys) + kFaKeys - 1) / kFaKeys;
        x.tiles = x.kept + (x.pos + x.count - 1) / kFaKeys - x.first + 1;
        x.pad = 0;
        return x;
    };
    for (int u = tid; u < units; u += 1024) atomicAdd(&bins[1023 - min(1023, unit_of(u).tiles)], 1);
    __syncthreads();
    const int mine = bins[tid], sum = scan(mine, true);
    __syncthreads();
    bins[tid] = sum - mine;
    __syncthreads();
    for (int u = tid; u < units; u += 1024) {
        const FlashUnit x = unit_of(u);
        flash_units(a)[atomicAdd(&bins[1023 - min(1023, x.tiles)], 1)] = x;
    }
    if (tid == 0) a.plan[0] = units;
}

// pieces of one block: the sorted list dealt out in turn, back and forth
struct FlashWalk {
    int lap, total;
    __device__ __forceinline__ explicit FlashWalk(const FlashArgs& a) : lap(0), total(a.plan[0] * a.kv_heads) {}
    __device__ __forceinline__ bool next(const FlashArgs& a, FlashUnit& x, int& head)
    {
        const int i = lap * gridDim.x + (lap & 1 ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
        ++lap;
        if (i >= total) return false;       // the later laps of this block lie further back still
        const int4* src = reinterpret_cast<const int4*>(flash_units(a) + i / a.kv_heads);
        const int4 u = src[0], v = src[1];
        x.row = u.x; x.count = u.y; x.pos = u.z; x.seq = u.w; x.first = v.x; x.kept = v.y; x.tiles = v.z;
        head = i % a.kv_heads;
        return true;
    }
};

// D: dimensions per map; MAPS * D columns of keys per position (64 or 128); V: value columns
template <int D, int MAPS, int V>
struct FlashShape {
    static constexpr int KC = D * MAPS;
    static constexpr int kQTile = 2 * 128 * D * 2;                // two bf16 parts of 128 rows
    static constexpr int kKTile = kFaKeys * KC * 2, kVTile = kFaKeys * V * 2;
    static constexpr int kStages = 2 * kQTile + 2 * (kKTile + kVTile) <= 224 * 1024 ? 2 : 1;
    static constexpr int kSmem = 2 * kQTile + kStages * (kKTile + kVTile);
};

// 16-byte units of 128 positions' rows of ROW bytes; a warp instruction takes 8 rows x 4 units, so that eight lanes store 128
// contiguous bytes of the operand tile [column / 8][position][8]
// Positions that no row of the unit sees (in front of the first row's window but not kept, or past the last row's) become zeros.
template <int ROW>
__device__ __forceinline__ void flash_fetch(const char* half0, const char* half1, int64_t stride, int key0, int lo, int keep, int last, unsigned dst, int w, int lane)
{
    constexpr int Q = ROW / 64, INSTR = kFaKeys / 8 * Q;
#pragma unroll
    for (int it = 0; it < (INSTR + kFaLoaders - 1) / kFaLoaders; ++it) {
        const int i = w + kFaLoaders * it;
        if (i >= INSTR) break;
        const int row = i / Q * 8 + (lane & 7), unit = i % Q * 4 + (lane >> 3);
        const bool in = key0 + row <= last && (key0 + row >= lo || key0 + row < keep);
        const char* src = (i / Q >= 8 ? half1 : half0) + (in ? (row & 63) * stride : 0) + unit * 16;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + unit * (kFaKeys * 16) + row * 16), "l"(src), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int D, int MAPS, int V>
__global__ void __launch_bounds__(kFaThreads, 1) flash_attention_kernel(const FlashArgs a)
{
    namespace umma = b200::umma;
    using b200::mbar_wait;
    using S = FlashShape<D, MAPS, V>;
    extern __shared__ __align__(1024) unsigned char fa_smem[];
    __shared__ uint64_t bar_q[2], bar_s[2], bar_p[4], bar_o[2];       // per tile: queries stored, scores ready, halves of the weights ready, values added
    __shared__ uint64_t bar_full[4], bar_empty[4];                     // rings of keys (0, 1) and of values (2, 3)
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = tid & 31;
    const int rep = a.heads / a.kv_heads, TQ = 128 / rep;             // heads per key/value head, tokens per tile
    if (warp == 8) umma::tmem_alloc(smem_u32(&s_tmem), 512);
    if (tid < 4) {
        if (tid < 2) {
            b200::mbar_init(smem_u32(&bar_q[tid]), 4);
            b200::mbar_init(smem_u32(&bar_s[tid]), 1);
            b200::mbar_init(smem_u32(&bar_o[tid]), 1);
        }
        b200::mbar_init(smem_u32(&bar_p[tid]), 4);
        b200::mbar_init(smem_u32(&bar_full[tid]), kFaLoaders);
        b200::mbar_init(smem_u32(&bar_empty[tid]), 1);
        b200::fence_mbar_init();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = s_tmem;                                      // columns: tile t's scores / weights at t * 128, accumulator at 256 + t * 128
    const uint32_t q_op = smem_u32(fa_smem), k_op = q_op + 2 * S::kQTile, v_op = k_op + S::kStages * S::kKTile;
    FlashWalk walk(a);
    FlashUnit x{};
    int head = 0;
    // tile t's tokens of the piece; its key tiles (a prefix of the piece's)
    auto tokens = [&](int t) { return MAPS == 2 ? x.count : max(0, min(TQ, x.count - t * TQ)); };
    auto tiles = [&](int t) {
        const int c = tokens(t);
        return c == 0 ? 0 : x.kept + (x.pos + (MAPS == 2 ? 0 : t * TQ) + c - 1) / kFaKeys - x.first + 1;
    };
    auto key_tile = [&](int i) { return i < x.kept ? i : i - x.kept + x.first; };

    if (warp > 8) {
        // ------------------------------------------------ loaders
        umma::set_max_registers_dec<64>();
        const int w = warp - 9;
        const int64_t k_row = (int64_t)a.kv_heads * S::KC * 2, v_row = (int64_t)a.kv_heads * V * 2;
        uint32_t count = 0, waiting = 0;
        auto publish = [&](uint32_t bar) {
            b200::fence_proxy_async();
            __syncwarp();
            if (lane == 0) b200::mbar_arrive(bar);
        };
        while (walk.next(a, x, head)) {
            const int64_t* pages = a.block_ptrs + a.cu_blocks[x.seq];
            const int last = x.pos + x.count - 1, lo = flash_lo(a, x.pos);
            // block_len is a multiple of 64: half a tile lies in one page
            auto find = [&](int i, const char*& p0, const char*& p1, int& o0, int& o1) {
                const int key = key_tile(i) * kFaKeys, b = key / a.block_len;
                p0 = reinterpret_cast<const char*>(pages[b]) + a.layer_off;
                o0 = key - b * a.block_len;
                p1 = p0; o1 = o0;
                if (key + 64 <= last) {
                    const int b1 = (key + 64) / a.block_len;
                    p1 = reinterpret_cast<const char*>(pages[b1]) + a.layer_off;
                    o1 = key + 64 - b1 * a.block_len;
                }
            };
            const char *p0, *p1, *n0, *n1;
            int o0, o1, m0, m1;
            find(0, p0, p1, o0, o1);
            for (int i = 0; i < x.tiles; ++i, ++count) {
                const uint32_t slot = count % S::kStages, ph = (count / S::kStages) & 1;
                n0 = p0; n1 = p1; m0 = o0; m1 = o1;
                if (i + 1 < x.tiles) find(i + 1, n0, n1, m0, m1);       // a tile ahead of its use
                const int key0 = key_tile(i) * kFaKeys;
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int bar = 8 * (2 * v + slot);
                    mbar_wait(smem_u32(&bar_empty[0]) + bar, ph ^ 1);
                    if (v == 0)
                        flash_fetch<S::KC * 2>(p0 + o0 * k_row + head * S::KC * 2, p1 + o1 * k_row + head * S::KC * 2, k_row, key0, lo, a.keep, last, k_op + slot * S::kKTile, w, lane);
                    else
                        flash_fetch<V * 2>(p0 + a.v_off + o0 * v_row + head * V * 2, p1 + a.v_off + o1 * v_row + head * V * 2, v_row, key0, lo, a.keep, last, v_op + slot * S::kVTile, w, lane);
                    if (S::kStages == 1) {                              // one slot: its own wait, or the ring would stand still
                        asm volatile("cp.async.wait_group 0;" ::: "memory");
                        publish(smem_u32(&bar_full[0]) + bar);
                    } else {
                        if (waiting) {
                            asm volatile("cp.async.wait_group 1;" ::: "memory");
                            publish(waiting);
                        }
                        waiting = smem_u32(&bar_full[0]) + bar;
                    }
                }
                p0 = n0; p1 = n1; o0 = m0; o1 = m1;
            }
            if (waiting) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                publish(waiting);
                waiting = 0;
            }
        }
    } else if (warp == 8) {
        // ------------------------------------------------ tensor-core products
        umma::set_max_registers_dec<64>();
        constexpr uint32_t kQk = umma::make_idesc_f16(128, kFaKeys, true), kPv = umma::make_idesc_f16(128, V, true) | (1u << 16);   // values: MN-major
        uint32_t count = 0, phq[2] = {0, 0}, php[2] = {0, 0};
        auto scores = [&](int t, uint32_t slot) {
            const uint64_t qd = umma::make_smem_desc(q_op + t * S::kQTile, 128 * 16, 128);
            const uint64_t kd = umma::make_smem_desc(k_op + slot * S::kKTile + (MAPS == 2 ? t * (D / 8) * (kFaKeys * 16) : 0), kFaKeys * 16, 128);
            if (b200::elect_one()) {
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks)
                        umma::mma_f16_ss(tmem + t * 128, qd + (uint64_t)((part * (D / 8) + 2 * ks) * (128 * 16) >> 4), kd + (uint64_t)(2 * ks * (kFaKeys * 16) >> 4), kQk,
                                         part > 0 || ks > 0);
                umma::commit(smem_u32(&bar_s[t]));
            }
            __syncwarp();
        };
        while (walk.next(a, x, head)) {
            const int n = x.tiles, cnt[2] = {tiles(0), tiles(1)};
            mbar_wait(smem_u32(&bar_full[count % S::kStages]), (count / S::kStages) & 1);
#pragma unroll
            for (int t = 0; t < 2; ++t)
                if (cnt[t] > 0) {
                    mbar_wait(smem_u32(&bar_q[t]), phq[t]);
                    phq[t] ^= 1;
                    umma::fence_after_sync();
                    scores(t, count % S::kStages);
                }
            if (b200::elect_one()) umma::commit(smem_u32(&bar_empty[count % S::kStages]));
            __syncwarp();
            for (int i = 0; i < n; ++i, ++count) {
                const uint32_t slot = count % S::kStages, ph = (count / S::kStages) & 1, next = (count + 1) % S::kStages, phn = ((count + 1) / S::kStages) & 1;
                mbar_wait(smem_u32(&bar_full[2 + slot]), ph);
                umma::fence_after_sync();
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (i < cnt[t]) {
                        const uint64_t vd = umma::make_smem_desc(v_op + slot * S::kVTile, 128, kFaKeys * 16);
#pragma unroll
                        for (int half = 0; half < 2; ++half) {          // the first 64 keys' products run under the second 64 keys' exponentials
                            mbar_wait(smem_u32(&bar_p[2 * half + t]), php[t]);
                            umma::fence_after_sync();
                            if (b200::elect_one()) {
#pragma unroll
                                for (int ks = 4 * half; ks < 4 * half + 4; ++ks)
#pragma unroll
                                    for (int part = 0; part < 2; ++part)
                                        umma::mma_f16_ts(tmem + 256 + t * 128, tmem + t * 128 + part * 64 + ks * 8, vd + (uint64_t)(ks * (256 >> 4)), kPv, i > 0 || ks > 0 || part > 0);
                                if (half) umma::commit(smem_u32(&bar_o[t]));
                            }
                            __syncwarp();
                        }
                        php[t] ^= 1;
                    }
                    if (t == 1 && b200::elect_one()) umma::commit(smem_u32(&bar_empty[2 + slot]));
                    __syncwarp();
                    if (i + 1 < n) {
                        if (t == 0) {
                            mbar_wait(smem_u32(&bar_full[next]), phn);
                            umma::fence_after_sync();
                        }
                        if (i + 1 < cnt[t]) scores(t, next);            // over the weights that the products just issued read: the pipe keeps the order
                        if (t == 1 && b200::elect_one()) umma::commit(smem_u32(&bar_empty[next]));
                        __syncwarp();
                    }
                }
            }
        }
    } else {
        // ------------------------------------------------ softmax: thread = row of tile t
        umma::set_max_registers_inc<192>();
        const int t = warp >> 2, r = tid & 127, tq = r / rep, g = r - tq * rep, map = MAPS == 2 ? t : 0;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16), ts = lanes + t * 128, to = lanes + 256 + t * 128;
        const float c = a.scale * 1.4426950408889634f;
        uint32_t phs = 0, pho = 0;
        auto arrive = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) b200::mbar_arrive(smem_u32(bar));
        };
        // the row's query as two bf16 parts -> [part][d / 8][row][8]; the products that read the earlier piece's have completed
        auto store_q = [&]() {
            if (tokens(t) == 0) return;
            const bool valid = tq < tokens(t);
            const float4* src = reinterpret_cast<const float4*>(a.qn + ((size_t)(x.row + (MAPS == 2 ? 0 : t * TQ) + tq) * a.heads * MAPS + (size_t)(head * rep + g) * MAPS + map) * D);
#pragma unroll 4
            for (int cc = 0; cc < D / 8; ++cc) {
                float4 f[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
                if (valid) { f[0] = src[2 * cc]; f[1] = src[2 * cc + 1]; }
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float u = (&f[k >> 1].x)[2 * (k & 1)], v = (&f[k >> 1].x)[2 * (k & 1) + 1];
                    hi[k] = b200::TypeOps<bf16>::pack2(u, v);
                    const float uh = __uint_as_float(hi[k] << 16), vh = __uint_as_float(hi[k] & 0xffff0000u);
                    lo[k] = b200::TypeOps<bf16>::pack2(isinf(uh) ? 0.f : u - uh, isinf(vh) ? 0.f : v - vh);
                }
                const uint32_t dst = q_op + t * S::kQTile + (cc * 128 + r) * 16;
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (D / 8) * 128 * 16), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
            }
            b200::fence_proxy_async();
            umma::fence_before_sync();
            arrive(&bar_q[t]);
        };
        bool more = walk.next(a, x, head);
        if (more) store_q();
        while (more) {
            const int nq = tokens(t), cnt = tiles(t), h = head * rep + g;
            const bool valid = tq < nq;
            const int pos0 = x.pos + (MAPS == 2 ? 0 : t * TQ), row = x.row + (MAPS == 2 ? 0 : t * TQ) + tq;
            const int pos = valid ? pos0 + tq : pos0, lo = flash_lo(a, pos), kept = min(a.keep, lo);       // padding rows do as the first row does
            const int lo_last = flash_lo(a, pos0 + max(nq, 1) - 1), first = x.first, front = x.kept;
            float m = -INFINITY, l = 0.f;
            for (int i = 0; i < cnt; ++i) {
                const int key0 = (i < front ? i : i - front + first) * kFaKeys;
                mbar_wait(smem_u32(&bar_s[t]), phs);
                phs ^= 1;
                umma::fence_after_sync();
                uint32_t v[4][32];
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) umma::ld_32x32b_x32(ts + ch * 32, v[ch]);
                umma::wait_ld();
                if (key0 + kFaKeys - 1 > pos0 || key0 < lo_last) {      // some row of the tile does not see some key
#pragma unroll
                    for (int k = 0; k < kFaKeys; ++k) {
                        const int j = key0 + k;
                        if (j > pos || (j < lo && j >= kept)) v[k >> 5][k & 31] = __float_as_uint(-INFINITY);
                    }
                }
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int k = 0; k < kFaKeys; ++k) mx4[k & 3] = fmaxf(mx4[k & 3], __uint_as_float(v[k >> 5][k & 31]));
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                if (i == 0) m = mx;
                else {
                    const float m_new = fmaxf(m, mx);
                    if (__any_sync(0xffffffffu, (m_new - m) * c > (float)kFaLazy)) {
                        const float alpha = m == -INFINITY ? 0.f : b200::exp2_approx((m - m_new) * c);
                        mbar_wait(smem_u32(&bar_o[t]), pho ^ 1);        // the previous tile's values have been added
                        umma::fence_after_sync();
#pragma unroll 1
                        for (int ch = 0; ch < V / 16; ++ch) {
                            uint32_t o[16];
                            umma::ld_32x32b_x16(to + ch * 16, o);
                            umma::wait_ld();
#pragma unroll
                            for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                            umma::st_32x32b_x16(to + ch * 16, o);
                        }
                        l *= alpha;
                        m = m_new;
                    }
                }
                const float mc = m == -INFINITY ? 0.f : m * c;
                float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int half = 0; half < 2; ++half) {
#pragma unroll
                    for (int ch = 2 * half; ch < 2 * half + 2; ++ch) {
                        uint32_t hi[16], low[16];                       // column c holds keys (2c, 2c + 1); the second parts 64 columns further
#pragma unroll
                        for (int k = 0; k < 32; k += 2) {
                            const float p0 = b200::exp2_approx(fmaf(__uint_as_float(v[ch][k]), c, -mc));
                            const float p1 = b200::exp2_approx(fmaf(__uint_as_float(v[ch][k + 1]), c, -mc));
                            l4[(k >> 1) & 3] += p0 + p1;
                            hi[k / 2] = b200::TypeOps<bf16>::pack2(p0, p1);
                            low[k / 2] = b200::TypeOps<bf16>::pack2(p0 - __uint_as_float(hi[k / 2] << 16), p1 - __uint_as_float(hi[k / 2] & 0xffff0000u));
                        }
                        umma::st_32x32b_x16(ts + ch * 16, hi);
                        umma::st_32x32b_x16(ts + 64 + ch * 16, low);
                    }
                    umma::wait_st();
                    umma::fence_before_sync();
                    arrive(&bar_p[2 * half + t]);
                }
                l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
                pho ^= 1;
            }
            // the next piece's query goes out before this one's output, so that its first scores are on their way meanwhile
            more = walk.next(a, x, head);
            if (more) store_q();
            if (cnt > 0) {
                mbar_wait(smem_u32(&bar_o[t]), pho ^ 1);
                umma::fence_after_sync();
            }
            // softmax denominator with the sink, as a factor on the accumulator
            float f = 1.0f / l;
            if (a.sink) {
                const float s = a.sink[h * MAPS + map] * 1.4426950408889634f, top = fmaxf(m * c, s);
                const float e = exp2f(m * c - top);
                f = e / (l * e + exp2f(s - top));
            }
            float* aside = MAPS == 2 ? a.second + ((size_t)row * a.heads + h) * V : nullptr;
            if (MAPS == 2 && t == 1) {
#pragma unroll 1
                for (int ch = 0; ch < V / 32; ++ch) {
                    uint32_t o[32];
                    umma::ld_32x32b_x32(to + ch * 32, o);
                    umma::wait_ld();
                    if (valid)
#pragma unroll
                        for (int k = 0; k < 8; ++k)
                            reinterpret_cast<float4*>(aside)[ch * 8 + k] = make_float4(__uint_as_float(o[4 * k]) * f, __uint_as_float(o[4 * k + 1]) * f,
                                                                                      __uint_as_float(o[4 * k + 2]) * f, __uint_as_float(o[4 * k + 3]) * f);
                }
            }
            if (MAPS == 2) b200::named_bar_sync(1, 256);                // the second map's outputs are in place (global, same block)
            if ((MAPS == 1 && cnt > 0) || (MAPS == 2 && t == 0)) {
                float norm = a.out_scale;
                auto columns = [&](int ch, float (&o)[32]) {
                    uint32_t raw[32];
                    umma::ld_32x32b_x32(to + ch * 32, raw);
                    umma::wait_ld();
#pragma unroll
                    for (int k = 0; k < 32; ++k) o[k] = __uint_as_float(raw[k]) * f;
                    if (MAPS == 2 && valid)
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const float4 s = reinterpret_cast<const float4*>(aside)[ch * 8 + k];
                            o[4 * k] -= a.lambda * s.x; o[4 * k + 1] -= a.lambda * s.y; o[4 * k + 2] -= a.lambda * s.z; o[4 * k + 3] -= a.lambda * s.w;
                        }
                };
                if (a.out_norm) {
                    float ss = 0.f;
#pragma unroll 1
                    for (int ch = 0; ch < V / 32; ++ch) {
                        float o[32];
                        columns(ch, o);
#pragma unroll
                        for (int k = 0; k < 32; ++k) ss = fmaf(o[k], o[k], ss);
                    }
                    norm = a.out_scale / sqrtf(ss / (float)V + a.eps);
                }
#pragma unroll 1
                for (int ch = 0; ch < V / 32; ++ch) {
                    float o[32];
                    columns(ch, o);
                    if (!valid) continue;
                    const int col = h * V + ch * 32;
                    const bf16* gate = a.gate ? a.gate + (size_t)row * a.ld_gate + col / a.gate_div : nullptr;
                    const float one = gate && a.gate_div > 1 ? sigmoid_f(to_f(gate[0])) : 1.0f;      // a gate per head
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint32_t z[4], out[4];
                        if (gate && a.gate_div == 1) {
                            const uint4 raw = *reinterpret_cast<const uint4*>(gate + 8 * k);
                            z[0] = raw.x; z[1] = raw.y; z[2] = raw.z; z[3] = raw.w;
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            float u = o[8 * k + 2 * q] * norm * one, w = o[8 * k + 2 * q + 1] * norm * one;
                            if (gate && a.gate_div == 1) {
                                u *= sigmoid_f(__uint_as_float(z[q] << 16));
                                w *= sigmoid_f(__uint_as_float(z[q] & 0xffff0000u));
                            }
                            out[q] = b200::TypeOps<bf16>::pack2(u, w);
                        }
                        *reinterpret_cast<uint4*>(a.y + (size_t)row * a.ld_y + col + 8 * k) = make_uint4(out[0], out[1], out[2], out[3]);
                    }
                }
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 8) umma::tmem_dealloc(tmem, 512);
}
