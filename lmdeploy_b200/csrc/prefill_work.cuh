// Prefill attention: how the work is cut and dealt out, as integers alone -- compiled by nvcc into the kernels of prefill_attention.cuh
// and by a host compiler into tests/test_prefill_work_cpu.py, which walks every CTA's list over many batches.
#pragma once

#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define B200_HD __host__ __device__ __forceinline__
#else
#define B200_HD inline
#endif

namespace b200 {
namespace attn {

constexpr int kPfRows    = 128;  // UMMA M: query rows per tile
constexpr int kPfKeys    = 128;  // keys per tile: UMMA N of S, K extent of P.V
constexpr int kPfD       = 128;
constexpr int kPfLoaders = 7;    // warps that fill the K/V rings
constexpr int kPfMaxCtas = 160;  // bound of the persistent grid (sizes the partial buffers)
constexpr int kPfStart   = 2;    // places that a piece takes in the work list before its key tiles (Q load, first scores, output)

#ifdef __CUDA_ARCH__
B200_HD int pf_min(int a, int b) { return min(a, b); }
B200_HD int pf_max(int a, int b) { return max(a, b); }
#else
B200_HD int pf_min(int a, int b) { return a < b ? a : b; }
B200_HD int pf_max(int a, int b) { return a > b ? a : b; }
#endif

struct alignas(16) PrefillUnit {
    int prefix;       // places of all earlier units in the work list (one kv-head): kPfStart, then one per 128-key tile
    int n;            // its own places
    int b, q0;        // sequence, first query token of the unit inside the chunk
    int tok0, q_len;  // the sequence's first token of the step and number of tokens
    int hist, pad;
};

// where a CTA's range of the work list begins, and the whole list's length; written by prefill_plan
struct alignas(16) PrefillRange {
    int u, r;       // unit, place inside it (all kv-heads)
    int count;      // places of the range
    int ctas;       // ranges in all
    long long total, pad;
};

struct PrefillParams {
    const void* q_rot;  // [token][Hq][D], bias + RoPE applied (prologue kernel)
    void*       out;    // [token][Hq*D]
    int64_t     out_stride;
    char**      block_ptrs;
    const int*  cu_block_nums;
    const int*  cu_q_len;
    const int*  cu_k_len;
    int         layer_offset;
    int         block_len;
    int         batch;
    int         num_heads;
    int         num_kv_heads;
    float       qk_scale;  // log2(e) / sqrt(D)
    PrefillUnit*  units;   // written by prefill_plan, one more than there are units
    PrefillRange* ranges;  // [main_ctas]
    int           main_ctas;
    float*       partial;  // [2 * CTA][2 tiles] partials, or null: whole (unit, kv-head) pieces are dealt out, without units and ranges
};

// tokens of a unit (two tiles), and its places in the work list
B200_HD int prefill_unit_tokens(const PrefillParams& p) { return 2 * (kPfRows / (p.num_heads / p.num_kv_heads)); }
B200_HD int prefill_places(int hist, int q_len, int q0, int TQ2) { return kPfStart + (hist + pf_min(q_len, q0 + TQ2) - 1) / kPfKeys + 1; }

// CTA c's range: equal numbers of places per CTA
B200_HD PrefillRange prefill_range(const PrefillParams& p, int n_units, int places, int c)
{
    const long long total = (long long)p.num_kv_heads * places;
    const int       ctas  = (int)(total < p.main_ctas ? total : p.main_ctas);
    PrefillRange    range{n_units, 0, 0, ctas, total, 0};
    if (c < ctas) {
        const long long at = total * c / ctas;
        int             lo = 0, hi = n_units;  // the last unit whose places (of all kv-heads) begin at or before `at`
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if ((long long)p.num_kv_heads * p.units[mid].prefix <= at) {
                lo = mid;
            }
            else {
                hi = mid;
            }
        }
        range.u     = lo;
        range.r     = (int)(at - (long long)p.num_kv_heads * p.units[lo].prefix);
        range.count = (int)(total * (c + 1) / ctas - at);
    }
    return range;
}

// One (unit, kv-head) piece: key tiles [j0, j1) of n
struct PrefillSegment {
    int b, q0, h, j0, j1, n;
    int q_len, hist, tok0;
    // tile t: valid query tokens and key tiles of it inside [j0, j1)
    B200_HD int tokens(int t, int TQ) const { return pf_max(0, pf_min(TQ, q_len - q0 - t * TQ)); }
    B200_HD int tiles(int t, int TQ) const
    {
        const int nq = tokens(t, TQ);
        return nq ? pf_max(0, pf_min(j1, (hist + q0 + t * TQ + nq - 1) / kPfKeys + 1) - j0) : 0;
    }
};

// walks the pieces of one CTA; every role of the CTA walks the same ones.  SPLIT: its range of the list; else whole pieces are dealt out in
// turn, without a list
template<bool SPLIT>
struct PrefillWalk;

template<>
struct PrefillWalk<true> {
    const PrefillParams& p;
    int                  u, r, left, n;  // unit, place inside it (all kv-heads), places left, the unit's places (0: not read yet)
    B200_HD PrefillWalk(const PrefillParams& p_, int cta): p(p_), n(0)
    {
        const PrefillRange range = p.ranges[cta];
        u = range.u, r = range.r, left = range.count;
    }
    // s: the piece that the last call gave
    B200_HD bool next(PrefillSegment& s)
    {
        do {
            if (left <= 0) {
                return false;
            }
            if (n > 0 && r >= p.num_kv_heads * n) {
                ++u, r = 0, n = 0;
            }
            if (n == 0) {
                const PrefillUnit unit = p.units[u];
                n = unit.n, s.n = unit.n - kPfStart;
                s.b = unit.b, s.q0 = unit.q0, s.tok0 = unit.tok0, s.q_len = unit.q_len, s.hist = unit.hist;
            }
            s.h            = r / n;
            const int from = r - s.h * n, to = pf_min(n, from + left);
            left -= to - from, r += to - from;
            s.j0 = pf_max(0, from - kPfStart);
            s.j1 = to - kPfStart;
        } while (s.j1 <= s.j0);  // the range holds no key tile of the piece
        return true;
    }
};

template<>
struct PrefillWalk<false> {
    const PrefillParams& p;
    int                  piece, b, before;  // next piece, its sequence or an earlier one, units of the sequences in front of that
    B200_HD PrefillWalk(const PrefillParams& p_, int cta): p(p_), piece(cta), b(0), before(0) {}
    B200_HD bool next(PrefillSegment& s)
    {
        const int TQ2 = prefill_unit_tokens(p), at = piece / p.num_kv_heads;
        for (;; ++b) {
            if (b >= p.batch) {
                return false;
            }
            s.tok0            = p.cu_q_len[b];
            s.q_len           = p.cu_q_len[b + 1] - s.tok0;
            const int n_units = (s.q_len + TQ2 - 1) / TQ2;
            if (at < before + n_units) {
                break;
            }
            before += n_units;
        }
        s.b    = b;
        s.q0   = (at - before) * TQ2;
        s.hist = p.cu_k_len[b + 1] - p.cu_k_len[b] - s.q_len;
        s.h    = piece % p.num_kv_heads;
        s.n    = prefill_places(s.hist, s.q_len, s.q0, TQ2) - kPfStart;
        s.j0 = 0, s.j1 = s.n;
        piece += p.main_ctas;
        return true;
    }
};

// where a CTA leaves its part of a piece: slot 0 if the piece began in an earlier CTA (its first one), else slot 1 (its last one)
B200_HD int prefill_slot(int cta, int j0) { return 2 * cta + (j0 > 0 ? 0 : 1); }

// The piece that CTA `first`'s range begins inside of, if that CTA is the second one with key tiles of it: whoever combines the parts
// asks every CTA but CTA 0 and finds each straddling piece once.
struct PrefillParts {
    PrefillUnit unit;
    int         h, cf, cl;  // kv-head, CTAs of the first and the last part
    // CTA cta's slot: only CTA cf's range begins at or before the piece
    B200_HD int slot(int cta) const { return 2 * cta + (cta == cf ? 1 : 0); }
};

B200_HD bool prefill_parts(const PrefillParams& p, int first, PrefillParts& x)
{
    const PrefillRange range = p.ranges[first];
    if (first >= range.ctas) {
        return false;
    }
    x.unit      = p.units[range.u];
    const int n = x.unit.n;
    x.h         = range.r / n;
    if (range.r - x.h * n <= kPfStart) {
        return false;  // the range begins with the piece
    }
    // the list's places of the piece's first and last key tile, and their CTAs (CTA c begins at place total * c / ctas)
    const long long s0 = (long long)p.num_kv_heads * x.unit.prefix + (long long)x.h * n + kPfStart, s1 = s0 + n - kPfStart - 1;
    x.cf = (int)(((s0 + 1) * range.ctas - 1) / range.total), x.cl = (int)(((s1 + 1) * range.ctas - 1) / range.total);
    return x.cf + 1 == first;  // else an earlier CTA has it
}

// Loader warps: the 16-byte units of 128 quantised token rows of K or of V.  A warp instruction takes 8 rows x 4 units (64 contiguous bytes per
// row); the 8 lanes that store one 8-dim chunk of as many rows write to eight places of a line's width (prefill_offset: no bank conflicts).
template<int KVBITS>
struct PrefillRowMap {
    static_assert(KVBITS == 8 || KVBITS == 4, "T rows: PrefillLineMap");
    static constexpr int kRow   = kPfD * KVBITS / 8;
    static constexpr int kUnits = kRow / 16;                               // 8 / 4 per row
    static constexpr int kInstr = kPfKeys / 8 * (kUnits / 4);              // warp instructions per tile
    static constexpr int kIter  = (kInstr + kPfLoaders - 1) / kPfLoaders;  // 5 / 3 per warp

    B200_HD static int key_of(int w, int lane, int it) { return (w + kPfLoaders * it) / (kUnits / 4) * 8 + (lane & 7); }
    B200_HD static int unit_of(int w, int lane, int it) { return (w + kPfLoaders * it) % (kUnits / 4) * 4 + (lane >> 3); }
    B200_HD static int half_of(int w, int it) { return (w + kPfLoaders * it) / (kUnits / 4) >> 3; }  // warp-uniform: key >> 6
};

// Operand tiles of Q, K and V: two halves of 64 dims, in each a row of 128 bytes per token whose 16-byte chunks are permuted by the row's last three
// bits (the tensor core's 128-byte swizzle).  So a row's line is stored as one line, and the same chunk of eight rows lies in eight places
// of a line's width.
B200_HD int prefill_offset(int chunk, int row) { return (chunk >> 3) * (kPfKeys * 128) + row * 128 + (((chunk & 7) ^ (row & 7)) << 4); }

// Loader warps: 128 rows of 256 bytes (T pages, queries).  A warp takes four rows at a time, two instructions of 4 rows x 128 bytes: eight consecutive
// lanes one line of both sides.
struct PrefillLineMap {
    static constexpr int kIter = (kPfKeys / 4 + kPfLoaders - 1) / kPfLoaders;  // 5 per warp

    B200_HD static bool inside(int w, int it) { return w + kPfLoaders * it < kPfKeys / 4; }
    B200_HD static int  row_of(int w, int lane, int it) { return (w + kPfLoaders * it) * 4 + (lane >> 3); }
    B200_HD static int  unit0(int lane) { return lane & 7; }  // of the first instruction; the second takes the unit eight behind
    // where row_of(w, lane, it), unit0(lane) lies in the operand tile: step(base + place(w, lane), it)
    B200_HD static uint32_t place(int w, int lane) { return (uint32_t)prefill_offset(unit0(lane), row_of(w, lane, 0)); }
    B200_HD static uint32_t step(uint32_t to, int it) { return (to ^ (it & 1 ? 64u : 0u)) + kPfLoaders * 512 * it; }  // 28 rows on: bit 2 of the row turns
};

}  // namespace attn
}  // namespace b200
