"""How prefill attention cuts and deals out its work (csrc/prefill_work.cuh, the header that the kernels compile), by a host compiler: over many ragged
batches, grids and GQA groups every key tile of every (sequence block, kv-head) is walked exactly once, the parts of a piece that CTAs share lie in the
slots that the merge reads, each by one CTA, and the form without room for partials walks the same pieces whole.  Also the loader warps' map of
quantised rows: every 16-byte unit of a tile once, every chunk of the operand tile once, eight lanes of a store in different banks."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "prefill_work.cuh"
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <set>
#include <tuple>
#include <vector>
using namespace b200::attn;

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s (case %d)\n", __LINE__, #x, g_case); std::exit(1); } } while (0)
static int g_case = 0;

struct Batch { std::vector<int> q, hist; };

static void run(const Batch& batch, int heads, int kv_heads, int grid, int order)
{
    ++g_case;
    std::vector<int> cu_q{0}, cu_k{0};
    for (size_t b = 0; b < batch.q.size(); ++b) cu_q.push_back(cu_q.back() + batch.q[b]), cu_k.push_back(cu_k.back() + batch.q[b] + batch.hist[b]);
    PrefillParams p{};
    p.cu_q_len = cu_q.data(), p.cu_k_len = cu_k.data();
    p.batch = (int)batch.q.size(), p.num_heads = heads, p.num_kv_heads = kv_heads, p.main_ctas = grid;
    // the list, in the order of the sequences
    std::vector<PrefillUnit> units;
    const int TQ2 = prefill_unit_tokens(p), TQ = TQ2 / 2;
    int places = 0;
    for (int b = 0; b < p.batch; ++b)
        for (int q0 = 0; q0 < batch.q[b]; q0 += TQ2) {
            const int n = prefill_places(batch.hist[b], batch.q[b], q0, TQ2);
            units.push_back(PrefillUnit{places, n, b, q0, cu_q[b], batch.q[b], batch.hist[b], 0});
            places += n;
        }
    const int n_units = (int)units.size();
    CHECK(n_units <= cu_q.back());                      // what the workspace holds
    units.push_back(PrefillUnit{places, 0, p.batch, 0, 0, 0, 0, 0});
    std::vector<PrefillRange> ranges(grid);
    p.units = units.data(), p.ranges = ranges.data();
    for (int c = 0; c < grid; ++c) ranges[c] = prefill_range(p, n_units, places, c);

    using Key = std::tuple<int, int, int>;              // sequence, first token, kv-head
    for (int split = 0; split < 2; ++split) {
        float room = 0;
        p.partial = split ? &room : nullptr;
        std::map<Key, std::vector<int>> seen;           // tiles walked, per piece
        std::map<Key, std::map<int, int>> parts;        // CTA -> slot
        std::set<int> slots;
        for (int c = 0; c < grid; ++c) {
            PrefillWalk<true>  w(p, c);
            PrefillWalk<false> v(p, c);
            PrefillSegment s;
            long long taken = 0;
            while (split ? w.next(s) : v.next(s)) {
                const int hist = batch.hist[s.b], q_len = batch.q[s.b];
                CHECK(s.q_len == q_len && s.hist == hist && s.tok0 == cu_q[s.b] && s.q0 % TQ2 == 0 && s.q0 < q_len && s.h >= 0 && s.h < kv_heads);
                const int last = hist + (q_len < s.q0 + TQ2 ? q_len : s.q0 + TQ2) - 1;
                CHECK(s.n == last / kPfKeys + 1 && s.j0 >= 0 && s.j0 < s.j1 && s.j1 <= s.n);
                for (int t = 0; t < 2; ++t) {           // a tile's rows: its own keys, no more
                    const int nq = s.tokens(t, TQ), want = nq ? (hist + s.q0 + t * TQ + nq - 1) / kPfKeys + 1 : 0;
                    const int hi = want < s.j1 ? want : s.j1;
                    CHECK(s.tiles(t, TQ) == (hi > s.j0 ? hi - s.j0 : 0));
                }
                CHECK(s.tiles(0, TQ) > 0 || s.j0 > 0);
                taken += s.j1 - s.j0;
                const Key key{s.b, s.q0, s.h};
                for (int j = s.j0; j < s.j1; ++j) seen[key].push_back(j);
                if (!(s.j0 == 0 && s.j1 == s.n)) {
                    CHECK(split);
                    const int slot = prefill_slot(c, s.j0);
                    CHECK(slot >= 0 && slot < 2 * kPfMaxCtas && slots.insert(slot).second);
                    parts[key][c] = slot;
                }
            }
            if (split) CHECK(taken <= ranges[c].count);
        }
        CHECK((int)seen.size() == n_units * kv_heads);
        for (auto& kv : seen) {
            auto v = kv.second;
            std::set<int> all(v.begin(), v.end());
            CHECK(all.size() == v.size() && *all.begin() == 0 && *all.rbegin() == (int)v.size() - 1);
            const int b = std::get<0>(kv.first), q0 = std::get<1>(kv.first);
            CHECK((int)v.size() == prefill_places(batch.hist[b], batch.q[b], q0, TQ2) - kPfStart);
        }
        if (!split) continue;
        std::set<Key> merged;
        for (int first = 1; first < grid; ++first) {
            PrefillParts x;
            if (!prefill_parts(p, first, x)) continue;
            const Key key{x.unit.b, x.unit.q0, x.h};
            CHECK(merged.insert(key).second && parts.count(key));
            auto& have = parts[key];
            CHECK((int)have.size() == x.cl - x.cf + 1 && x.cl < grid);
            for (int c = x.cf; c <= x.cl; ++c) CHECK(have.count(c) && have[c] == x.slot(c));
        }
        CHECK(merged.size() == parts.size());
    }
}

template<int KVBITS>
static void rows()
{
    using M = PrefillRowMap<KVBITS>;
    std::set<int> units, places;
    for (int w = 0; w < kPfLoaders; ++w)
        for (int it = 0; it < M::kIter; ++it) {
            if (w + kPfLoaders * it >= M::kInstr) break;
            for (int lane = 0; lane < 32; ++lane) {
                const int key = M::key_of(w, lane, it), unit = M::unit_of(w, lane, it);
                CHECK(key >= 0 && key < kPfKeys && unit >= 0 && unit < M::kUnits && M::half_of(w, it) == key / 64);
                CHECK(units.insert(key * M::kUnits + unit).second);
                for (int k = 0; k < 16 / KVBITS; ++k) CHECK(places.insert(prefill_offset(unit * (16 / KVBITS) + k, key)).second);
            }
            for (int k = 0; k < 16 / KVBITS; ++k)        // eight lanes store at once, each to 16 bytes of its own among the 32 banks
                for (int group = 0; group < 4; ++group) {
                    std::set<int> banks;
                    for (int lane = 8 * group; lane < 8 * group + 8; ++lane)
                        banks.insert(prefill_offset(M::unit_of(w, lane, it) * (16 / KVBITS) + k, M::key_of(w, lane, it)) / 16 % 8);
                    CHECK(banks.size() == 8);
                }
        }
    CHECK((int)units.size() == kPfKeys * M::kUnits && (int)places.size() == kPfKeys * kPfD / 8);
    CHECK(*places.begin() == 0 && *places.rbegin() + 16 == kPfKeys * kPfD * 2);
}

int main(int argc, char** argv)
{
    std::mt19937 rng(std::atoi(argv[1]));
    auto pick = [&](int n) { return (int)(rng() % n); };
    rows<8>(), rows<4>();
    const int heads[][2] = {{32, 8}, {48, 8}, {64, 8}, {28, 4}, {16, 8}, {8, 2}, {7, 1}, {2, 2}, {128, 1}, {3, 1}, {100, 1}};
    const int edges[] = {0, 1, 2, 63, 64, 65, 127, 128, 129, 255, 256, 257, 383, 384};
    for (int i = 0; i < 4000; ++i) {
        Batch batch;
        const int n = 1 + (i % 3 ? pick(9) : 0);
        for (int b = 0; b < n; ++b) {
            const int kind = pick(4);
            batch.q.push_back(kind == 0 ? edges[pick(14)] : kind == 1 ? 1 : 1 + pick(kind == 2 ? 40 : 700));
            batch.hist.push_back(pick(3) == 0 ? edges[pick(14)] : pick(3) ? pick(300) : pick(9000));
        }
        const auto& h = heads[pick(11)];
        const int grids[] = {148, 160, 1, 2, 3, 1 + pick(160)};
        run(batch, h[0], h[1], grids[pick(6)], i);
    }
    std::printf("ok %d\n", g_case);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("prefill_work")
    (d / "main.cpp").write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "lmdeploy_b200", "csrc"), str(d / "main.cpp"), "-o", str(d / "main")], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    return str(d / "main")


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_every_key_tile_is_walked_once_and_every_part_found(program, seed):
    r = subprocess.run([program, str(seed)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
