// The warp's beam on the host (host_warp.hpp) against plain sorted lists: insertion and
// choice of the next entry, and whole searches, with finite distances, infinities and
// NaN (farther than everything, equal to each other).  Prints what differs; exit 1.
#include "host_warp.hpp"

#include <algorithm>
#include <deque>
#include <random>
#include <set>

#include "../hrnn_b200/csrc/beam.cuh"
#include "../hrnn_b200/csrc/beam_fast.cuh"

using namespace hrnn;

namespace {

std::mt19937 rng(7);
const float kNan = NAN, kInf = INFINITY;

unsigned pick(unsigned n) { return (unsigned)(rng() % n); }
bool nearer(float a, float b) { return std::isnan(b) ? !std::isnan(a) : a < b; }
bool same(float a, float b) { return a == b || (std::isnan(a) && std::isnan(b)); }

struct Entry {
    float d;
    uint32_t id;
    bool expanded;
};

// The reference's sequential rule: a neighbour that is not in the beam enters it while
// there is room or the last entry is farther.
struct Plain {
    std::vector<Entry> e;
    size_t EF;
    void add(float d, uint32_t id) {
        for (const Entry& x : e)
            if (x.id == id) return;
        if (e.size() >= EF && !nearer(d, e.back().d)) return;
        auto at = std::find_if(e.begin(), e.end(), [&](const Entry& x) { return nearer(d, x.d); });
        e.insert(at, Entry{d, id, false});
        if (e.size() > EF) e.pop_back();
    }
    size_t first() const {
        return (size_t)(std::find_if(e.begin(), e.end(), [](const Entry& x) { return !x.expanded; }) - e.begin());
    }
};

std::vector<char> pool(1 << 20);
char* smem() {
    std::memset(pool.data(), 0x5A, pool.size());  // what a kernel finds there
    return (char*)(((uintptr_t)pool.data() + 63) & ~(uintptr_t)63);
}

int bad(const char* what, const WarpSmem& s, uint32_t n, const Plain& p) {
    std::printf("%s: EF %zu, %u entries for %zu\n", what, p.EF, n, p.e.size());
    for (size_t i = 0; i < std::max<size_t>(n, p.e.size()) && i < 40; ++i)
        std::printf("  %zu: %g %u | %g %u\n", i, i < n ? s.td[i] : 0.f, i < n ? s.ti[i] : 0u,
                    i < p.e.size() ? p.e[i].d : 0.f, i < p.e.size() ? p.e[i].id : 0u);
    return 1;
}

bool equal(const WarpSmem& s, uint32_t n, const Plain& p) {
    if (n != p.e.size()) return false;
    for (uint32_t i = 0; i < n; ++i)
        if (!same(s.td[i], p.e[i].d) || s.ti[i] != (p.e[i].id | (p.e[i].expanded ? kExpanded : 0u))) return false;
    return true;
}

// Steps of a search with made-up neighbours whose distances come from `values`.
template <bool DEDUP>
int insertion(uint32_t EF, const std::vector<float>& values, bool exact) {
    const uint32_t ids = 400;
    std::vector<float> dist(ids);
    for (float& d : dist) d = values[pick((unsigned)values.size())];
    const uint32_t efc = (EF + 31) & ~31u;
    WarpSmem s = carve(smem(), 16, efc, 256);
    Plain p;
    p.EF = EF;
    p.add(dist[0], 0);
    s.td[0] = dist[0];
    s.ti[0] = 0;
    uint32_t tsize = 1, cursor = 0;
    for (int step = 0; step < 60; ++step) {
        const size_t f = p.first();
        if (f == p.e.size()) break;
        p.e[f].expanded = true;
        s.ti[f] |= kExpanded;
        cursor = (uint32_t)f + 1;
        const uint32_t cnt = pick(33);
        std::vector<uint32_t> nb;
        while (nb.size() < cnt) {
            const uint32_t id = pick(ids);
            if (DEDUP || std::find(nb.begin(), nb.end(), id) == nb.end()) nb.push_back(id);
        }
        uint32_t size[32], cur[32], next[32], place[32];
        std::fill(next, next + 32, kInvalid - 1);
        if (!hostwarp::run(
                [&] {
                    const uint32_t lane = threadIdx.x;
                    uint32_t n = tsize, c = cursor, at = 0;
                    const uint32_t after = first_unexpanded(s, c, n, at);
                    const bool have = lane < cnt;
                    beam_insert<DEDUP>(s, have ? dist[nb[lane]] : 0.f, have ? nb[lane] : kInvalid, have, EF, n, c,
                                       [&](float d, bool ok, uint32_t id, uint32_t pos) {
                                           if (!exact) return;
                                           next[lane] = next_entry(s, d, ok, id, pos, after, at);
                                           place[lane] = at;
                                       });
                    size[lane] = n;
                    cur[lane] = c;
                },
                100000))
            return std::printf("an insertion does not end\n"), 1;
        tsize = size[0];
        cursor = cur[0];
        for (uint32_t id : nb) p.add(dist[id], id);
        if (!equal(s, tsize, p)) return bad("insertion", s, tsize, p);
        const size_t g = p.first();
        for (size_t i = 0; i < std::min<size_t>(cursor, p.e.size()); ++i)
            if (!p.e[i].expanded) return bad("cursor", s, tsize, p);
        if (exact) {
            const uint32_t want = g < p.e.size() ? p.e[g].id : kInvalid;
            if (next[0] != want || (want != kInvalid && place[0] != g)) {
                std::printf("next %u at %u, not %u at %zu\n", next[0], place[0], want, g);
                return bad("next entry", s, tsize, p);
            }
        }
    }
    return 0;
}

// Searches of a random graph of n points with one coordinate each, deg links a point.
struct Graph {
    std::vector<float> x;
    std::vector<uint16_t> bf;
    std::vector<uint32_t> adj;
    DevView v{};
    Graph(uint32_t n, uint32_t deg, const std::vector<float>& values, float finite) : x(n), bf(n), adj((size_t)n * (deg + 1)) {
        for (uint32_t i = 0; i < n; ++i) {
            x[i] = pick(1000) < 1000 * finite ? 1.f + 1e-3f * (float)pick(4096) : values[pick((unsigned)values.size())];
            bf[i] = (uint16_t)(__float_as_uint(x[i]) >> 16);
            uint32_t* row = &adj[(size_t)i * (deg + 1)];
            row[0] = deg;
            for (uint32_t j = 1; j <= deg;) {
                row[j] = pick(n);
                if (std::find(row + 1, row + j, row[j]) == row + j && row[j] != i) ++j;
            }
        }
        v.vec = x.data();
        v.vec_bf16 = bf.data();
        v.adj0 = adj.data();
        v.n = n;
        v.dim = 1;
        v.W0 = deg + 1;
        v.lanes = 16;
    }
};

int exact_search(const Graph& g, float q, uint32_t EF, uint32_t vc) {
    const uint32_t deg = g.v.W0 - 1, efc = (EF + 31) & ~31u;
    auto dist = [&](uint32_t i) { return (q - g.x[i]) * (q - g.x[i]); };
    Plain p;
    p.EF = EF;
    p.add(dist(0), 0);
    std::set<uint32_t> met{0};
    unsigned long long want = 0;
    for (size_t f; (f = p.first()) < p.e.size(); ++want) {
        p.e[f].expanded = true;
        const uint32_t c = p.e[f].id;
        for (uint32_t j = 0; j < deg; ++j) {
            const uint32_t id = g.v.adj0[(size_t)c * (deg + 1) + 1 + j];
            if (met.insert(id).second) p.add(dist(id), id);
        }
    }
    WarpSmem s = carve(smem(), 1, efc, vc);
    s.q[0] = q;
    uint32_t size[32];
    unsigned long long exp[32];
    if (!hostwarp::run(
            [&] {
                unsigned long long nd = 0, ne = 0;
                size[threadIdx.x] = beam_search<0, kRowsAny>(g.v, s, 0, dist(0), EF, 0, vc, nd, ne);
                exp[threadIdx.x] = ne;
            },
            2000000))
        return std::printf("a search (EF %u, %u slots, %u links) does not end\n", EF, vc, deg), 1;
    if (!equal(s, size[0], p)) return bad("search", s, size[0], p);
    if (exp[0] != want) return std::printf("%llu expansions, not %llu\n", exp[0], want), 1;
    return 0;
}

int fast_search(const Graph& g, float q, uint32_t EF, uint32_t vc) {
    WarpSmem s = carve_fast(smem(), 16, (EF + 31) & ~31u, vc);
    s.q[0] = q;
    uint32_t size[32];
    if (!hostwarp::run(
            [&] {
                const uint32_t lane = threadIdx.x;
                unsigned long long nd = 0, ne = 0;
                for (uint32_t i = lane; i < vc; i += 32) s.vis[i] = kInvalid;
                if (lane == 0) {
                    s.td[0] = bf16_thread(s.q, g.v.vec_bf16, 1);
                    s.ti[0] = 0;
                }
                __syncwarp();
                size[lane] = beam_search_fast<2, false, 0>(g.v, s, 1, EF, EF, vc, nd, ne);
            },
            2000000))
        return std::printf("a two-parent search does not end\n"), 1;
    std::set<uint32_t> ids;
    for (uint32_t i = 0; i < size[0]; ++i) {
        const uint32_t id = s.ti[i] & kIdMask;
        if (id >= g.v.n || !ids.insert(id).second || !same(s.td[i], bf16_thread(s.q, g.v.vec_bf16 + id, 1)) ||
            (i && nearer(s.td[i], s.td[i - 1])))
            return std::printf("two-parent beam: entry %u is %u, %g\n", i, id, s.td[i]), 1;
    }
    return 0;
}

// The descent through two upper levels of a random graph, lists of `deg` links.
int descent(uint32_t n, uint32_t deg, const std::vector<float>& values, float finite, float q) {
    Graph g(n, 16, values, finite);
    std::vector<uint32_t> up;
    std::vector<uint64_t> off(n);
    for (uint32_t i = 0; i < n; ++i) {
        off[i] = up.size();
        for (int level = 0; level < 2; ++level) {
            up.push_back(pick(8) ? deg : pick(deg + 1));
            for (uint32_t j = 0; j < deg; ++j) up.push_back(pick(n));
        }
    }
    g.v.upper = up.data();
    g.v.upper_off = off.data();
    g.v.WU = deg + 1;
    auto dist = [&](uint32_t i) { return (q - g.x[i]) * (q - g.x[i]); };
    uint32_t want = 0;
    for (int level = 2; level > 0; --level)
        for (bool moved = true; moved;) {
            moved = false;
            const uint32_t* row = &up[off[want] + (size_t)(level - 1) * (deg + 1)];
            uint32_t best = want;
            for (uint32_t j = 0; j < row[0]; ++j)
                if (dist(row[1 + j]) < dist(best)) {
                    best = row[1 + j];
                    moved = true;
                }
            want = best;
        }
    WarpSmem s = carve(smem(), 1, 32, 256);
    s.q[0] = q;
    uint32_t got[32];
    if (!hostwarp::run(
            [&] {
                unsigned long long nd = 0;
                uint32_t cur = 0;
                float curd = dist(0);
                greedy_descent<0, kRowsAny>(g.v, s, 2, 0, cur, curd, nd);
                got[threadIdx.x] = cur;
            },
            1000000))
        return std::printf("a descent does not end\n"), 1;
    if (got[0] != want) return std::printf("descent to %u, not %u (query %g)\n", got[0], want, q), 1;
    return 0;
}

// A link list's candidates by (distance, id).
int candidates(uint32_t n, const std::vector<float>& values) {
    std::vector<uint32_t> id(n);
    std::vector<float> d(n);
    for (uint32_t i = 0; i < n; ++i) {
        id[i] = (i * 7919u) % 4099u;
        d[i] = values[pick((unsigned)values.size())];
    }
    std::vector<uint32_t> at(n);
    for (uint32_t i = 0; i < n; ++i) at[i] = i;
    std::sort(at.begin(), at.end(), [&](uint32_t a, uint32_t b) {
        return nearer(d[a], d[b]) || (same(d[a], d[b]) && id[a] < id[b]);
    });
    std::vector<uint64_t> keys(n, ~0ull);
    if (!hostwarp::run([&] { order_candidates(id.data(), d.data(), n, keys.data()); }, 1000))
        return std::printf("an ordering does not end\n"), 1;
    for (uint32_t i = 0; i < n; ++i)
        if ((uint32_t)keys[i] != id[at[i]] || !same(__uint_as_float((uint32_t)(keys[i] >> 32)), d[at[i]]))
            return std::printf("candidate %u of %u: %u, not %u\n", i, n, (uint32_t)keys[i], id[at[i]]), 1;
    return 0;
}

}  // namespace

int main() {
    const std::vector<std::vector<float>> kinds = {
        {0.f, .25f, .5f, 1.f, 2.f, 3.f, 4.f, 1e30f}, {kNan}, {kInf}, {0.f, 1.f, 2.f, kNan}, {0.f, 1.f, kInf, kNan},
        {kInf, kNan}};
    int r = 0;
    for (const auto& k : kinds)
        for (uint32_t EF : {1u, 2u, 31u, 32u, 33u, 64u, 130u, 300u})
            for (int t = 0; t < 6 && !r; ++t) {
                r = insertion<false>(EF, k, true) || insertion<true>(EF, k, false);
                auto signs = k;  // INT8 forms: a distance near 0 may come out negative
                signs.push_back(-1.f);
                r = r || insertion<true>(EF, signs, false);
            }
    for (const auto& k : kinds)
        for (float finite : {0.f, .9f})
            for (uint32_t deg : {16u, 32u, 40u}) {
                if (r) break;
                const Graph g(1200, deg, k, finite);
                for (uint32_t EF : {1u, 150u})
                    for (uint32_t vc : {256u, 512u})
                        for (float q : {0.f, 2.5f, kNan})
                            if (!r) r = exact_search(g, q, EF, vc) || (deg <= 32 && fast_search(g, q, EF, vc));
            }
    for (const auto& k : kinds)
        for (uint32_t n : {1u, 17u, 33u, 300u})
            if (!r) r = candidates(n, k);
    for (const auto& k : kinds)
        for (float finite : {0.f, .5f, 1.f})
            for (uint32_t deg : {3u, 16u, 32u, 40u})
                for (float q : {0.f, 2.5f, kNan, kInf, 1e30f})
                    if (!r) r = descent(300, deg, k, finite, q);
    return r;
}
