// Batched HNSW insertion on the device: the addPoint loop of hrnn_build
// (src/hrnn_build.cpp:75-88; addPoint hrnn.h:1378-1517) with the KNN-graph seed
// of hrnn.h:1479-1501.
//
// Points are inserted in batches that grow with the index (1/24 of the current
// size, at most 16384 points) and are all enqueued without a wait.  For every point of
// a batch one warp, or a team of warps while batches are small, runs against the
// graph as it was at the start of the batch:
//   - the greedy descent from the entry point down to the point's level + 1;
//   - per level l <= min(level, maxlevel): the ef_construction beam search of
//     that layer (beam.cuh), the KNN-graph seed at level 0 (the beam, ascending,
//     self excluded, at most K entries), and the neighbour heuristic
//     getNeighborsByHeuristic2 (hrnn.h:619-659) choosing at most M links, written
//     in the reference's order (farthest first, hrnn.h:695-699) -- the nearest
//     link is the entry point of the next level (hrnn.h:700);
//   - one link back (target list, new point, distance) per link, into the target
//     list's slots.
// Then k_link_update applies all links back of the batch, one warp per target
// list: new points are appended while the list has room, otherwise the union of
// the list and the new points is pruned with the same heuristic to maxM0 (level
// 0) or maxM links (mutuallyConnectNewElement, hrnn.h:729-797).
//
// Levels come from the reference's generator in insertion order
// (getRandomLevel, hrnn.h:383-387; std::default_random_engine seeded with
// random_seed).  Points of one batch do not see each other while searching; the
// graph therefore differs from a sequential build (as the reference's own
// multi-threaded build does), while every stored distance is the exact FP32 value
// of the reference's L2 order.
#include <algorithm>
#include <cstdlib>
#include <cfloat>
#include <cmath>
#include <random>
#include <vector>

#include "beam.cuh"
#include "index.hpp"

namespace hrnn {

DevView make_view(Index& ix);

namespace {

// Reverse links asked for by a batch, by target list (`key`: node id for level 0,
// cap + upper block index above).  Every link has a number of its own below maxreq; the
// first to come to a list gives it its record, so only 8 bytes per list are needed
// (40 with a record per list: 320 MB for one point inserted into an index with room for
// 8M).  The first kSlots of a list sit in its record; further ones (lists of hub points)
// are chained from the record's head, each in its number's place.  The new points are
// sorted before they are used, so no grouping pass is needed, and the order of arrival
// matters only for a list with more than kGroupMax links of one batch: it decides which
// of them are applied, the others are dropped.
struct Link {
    uint32_t src;     // new point
    float d;          // L2(new point, target)
};
constexpr uint32_t kSlots = 4;
struct OverLink {
    Link l;
    uint32_t next;    // kInvalid ends the chain
};
struct ListLinks {
    uint32_t cnt;     // links asked for
    uint32_t rec;     // 1 + the list's record (0: none yet)
};
struct ActiveList {
    uint32_t key, target, rec;  // target: the node the list is of
};
struct LinkTable {
    ListLinks* list;      // [keys] zeros between batches
    uint32_t* head;       // [maxreq] a record's latest chained link (kInvalid between batches)
    Link* slot;           // [maxreq][kSlots]
    OverLink* over;       // [maxreq]
    ActiveList* active;   // [maxreq] the lists with new links
    uint32_t* ctr;        // this batch's counters: active lists, links above level 0
};

constexpr uint32_t kMaxSel = 64;      // M of the heuristic (maxM0 for reverse pruning)
constexpr uint32_t kGroupMax = 1024;  // new links applied to one list per batch

// Heuristic of hrnn.h:619-659 on a candidate list sorted by distance to the base
// point: keep a candidate unless a kept one is closer to it than the base is, until
// M are kept.
//
// The candidates are taken in blocks that sit in registers (dim = 16 NB, four lanes
// per row as in warp_l2_quads, G groups of eight rows): the block's live candidates
// are tested against the kept ones in the order these were kept, and when they have
// met all of them the first live candidate is kept and its row written to rows[]
// (shared memory, nfit rows; later ones are read from global memory).  Testing
// candidate by candidate, each with its own two dependent global reads, made this
// half of a construction search.
template <bool FUSED, int NB, int G>
__device__ uint32_t heuristic_block(const DevView& v, const uint32_t* cid, const float* cdist, uint32_t nc, uint32_t M,
                                    float* rows, uint32_t nfit, uint32_t* sel_id, float* sel_d) {
    constexpr uint32_t dim = 16 * NB;
    const int lane = threadIdx.x & 31, c = lane & 3, r = lane >> 2;
    uint32_t ns = 0;
    for (uint32_t base = 0; base < nc && ns < M; base += 8 * G) {
        float4 x[G][NB];
        float dq[G];
        bool live[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint32_t t = base + 8 * g + r;
            live[g] = t < nc;
            dq[g] = cdist[live[g] ? t : base];
            const float4* x4 = reinterpret_cast<const float4*>(v.vec + (size_t)cid[live[g] ? t : base] * dim) + c;
#pragma unroll
            for (int i = 0; i < NB; ++i) x[g][i] = __ldg(x4 + 4 * i);
        }
        for (uint32_t met = 0;;) {
            uint32_t alive[G], any = 0;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                alive[g] = __ballot_sync(0xFFFFFFFFu, live[g]);
                any |= alive[g];
            }
            if (!any) break;
            if (met == ns) {  // every kept one is farther: keep the first live candidate
                bool taken = false;
#pragma unroll
                for (int g = 0; g < G; ++g)
                    if (!taken && alive[g]) {
                        taken = true;
                        const int rr = (__ffs(alive[g]) - 1) >> 2;
                        if (r == rr) {
                            live[g] = false;
                            if (ns < nfit) {
                                float4* dst = reinterpret_cast<float4*>(rows + (size_t)ns * dim) + c;
#pragma unroll
                                for (int i = 0; i < NB; ++i) dst[4 * i] = x[g][i];
                            }
                            if (c == 0) {
                                sel_id[ns] = cid[base + 8 * g + r];
                                sel_d[ns] = dq[g];
                            }
                        }
                    }
                __syncwarp();
                if (++ns == M) break;
            }
            // the live candidates against kept row `met`
            const float4* s4 =
                reinterpret_cast<const float4*>(met < nfit ? rows + (size_t)met * dim : v.vec + (size_t)sel_id[met] * dim) + c;
            float acc[G][4];
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[g][k] = 0.f;
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const float4 p = s4[4 * i];
#pragma unroll
                for (int g = 0; g < G; ++g) quad_step<FUSED>(acc[g], p, x[g][i]);
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const float d = quad_sum16(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
                if (d < dq[g]) live[g] = false;
            }
            ++met;
        }
    }
    __syncwarp();
    return ns;
}

// The same with the live candidates of a 32-candidate block as a list, for the
// other dims and orders.  ids (32) and dl (32): scratch in shared memory.
template <bool FUSED, int RK>
__device__ uint32_t heuristic_list(const DevView& v, const uint32_t* cid, const float* cdist, uint32_t nc, uint32_t M,
                                   uint32_t* sel_id, float* sel_d, uint32_t* ids, float* dl) {
    const int lane = threadIdx.x & 31;
    uint32_t ns = 0;
    for (uint32_t base = 0; base < nc && ns < M; base += 32) {
        bool live = base + lane < nc;
        const uint32_t id = cid[live ? base + lane : base];
        const float dq = cdist[live ? base + lane : base];
        for (uint32_t met = 0;;) {
            uint32_t alive = __ballot_sync(0xFFFFFFFFu, live);
            if (!alive) break;
            if (met == ns) {
                const int first = __ffs(alive) - 1;
                if (lane == first) {
                    live = false;
                    sel_id[ns] = id;
                    sel_d[ns] = dq;
                }
                __syncwarp();
                if (++ns == M) break;
                alive &= alive - 1;
                if (!alive) break;
            }
            const uint32_t at = __popc(alive & lanemask_lt());
            if (live) ids[at] = id;
            __syncwarp();
            warp_l2_list<FUSED, RK>(v, v.vec + (size_t)sel_id[met] * v.dim, ids, __popc(alive), dl);
            if (live && dl[at] < dq) live = false;
            __syncwarp();
            ++met;
        }
    }
    return ns;
}

// rows: shared-memory room for nfit vectors; scratch: 64 words.  Returns the number
// kept (all candidates when fewer than M).
template <bool FUSED, int RK>
__device__ uint32_t heuristic(const DevView& v, const uint32_t* cid, const float* cdist, uint32_t nc, uint32_t M,
                              float* rows, uint32_t nfit, uint32_t* sel_id, float* sel_d, uint32_t* scratch) {
    const int lane = threadIdx.x & 31;
    if (nc < M) {
        for (uint32_t i = lane; i < nc; i += 32) {
            sel_id[i] = cid[i];
            sel_d[i] = cdist[i];
        }
        __syncwarp();
        return nc;
    }
    if constexpr (RK >= 64)
        return heuristic_block<FUSED, RK / 16, RK <= 128 ? 2 : 1>(v, cid, cdist, nc, M, rows, nfit, sel_id, sel_d);
    else
        return heuristic_list<FUSED, RK>(v, cid, cdist, nc, M, sel_id, sel_d, scratch, (float*)(scratch + 32));
}

// Shared memory of one k_build_batch warp.
__host__ __device__ inline size_t build_warp_bytes(uint32_t dim, uint32_t efc, uint32_t vc) {
    return (warp_smem_bytes(dim, efc, vc) + kMaxSel * 8 + 64 * 4 + 15) & ~(size_t)15;
}

// T: warps per point.  1: a warp of its own for each point, four to a block.
// kTeamWarps: the block's warps search for one point (beam_search_team) and warp 0
// does the rest, for batches too small to fill the device.
template <bool FUSED, int RK, int T>
__global__ void __launch_bounds__(T == 1 ? 128 : 32 * T, T == 1 ? 4 : 2) k_build_batch(DevView v, uint32_t b0, uint32_t b1, uint32_t ep, int maxlevel,
                                                        uint32_t efc, uint32_t vc, uint32_t M, uint32_t cap,
                                                        const int32_t* __restrict__ levels, uint32_t K,
                                                        uint32_t* __restrict__ knn_hdr, uint32_t* __restrict__ knn_ids,
                                                        float* __restrict__ knn_dist, uint32_t* __restrict__ adj0,
                                                        uint32_t* __restrict__ upper, LinkTable lt) {
    extern __shared__ __align__(16) char smem_raw[];
    constexpr int DM = FUSED ? 1 : 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const uint32_t ut = T == 1 ? lane : threadIdx.x, un = 32 * T;  // thread within the point's warps
    char* base = smem_raw + (T == 1 ? (size_t)w * build_warp_bytes(v.dim, efc, vc) : 0);
    WarpSmem s = carve(base, v.dim, efc, vc);
    uint32_t* sel_id = (uint32_t*)(base + warp_smem_bytes(v.dim, efc, vc));
    float* sel_d = (float*)(sel_id + kMaxSel);
    uint32_t* scratch = (uint32_t*)(sel_d + kMaxSel);
    auto sync = [] {
        if constexpr (T == 1) __syncwarp();
        else __syncthreads();
    };
    unsigned long long c_dist = 0, c_exp = 0;
    const uint32_t stride = T == 1 ? gridDim.x * wpb : gridDim.x;
    for (uint32_t p = b0 + (T == 1 ? blockIdx.x * wpb + w : blockIdx.x); p < b1; p += stride) {
        for (uint32_t i = ut; i < v.dim; i += un) s.q[i] = v.vec[(size_t)p * v.dim + i];
        sync();
        const int L = levels[p];
        uint32_t cur = ep;
        float curd = 0.f;
        if (T == 1 || w == 0) {
            curd = warp_dist_one<DM, RK>(v, s.q, cur);
            if (L < maxlevel) greedy_descent<DM, RK>(v, s, maxlevel, L, cur, curd, c_dist);  // hrnn.h:1438-1464
        }
        for (int level = min(L, maxlevel); level >= 0; --level) {
            if constexpr (T > 1) __syncthreads();  // warp 0 is done with the level above
            uint32_t tsize;
            if constexpr (T == 1) {
                tsize = beam_search<DM, RK>(v, s, cur, curd, efc, level, vc, c_dist, c_exp);
            } else {
                // (warp 0's cur and curd reach the others through the beam's first entry)
                tsize = efc <= 256 ? beam_search_team<FUSED, RK, 8>(v, s, scratch, cur, curd, efc, level, vc, c_dist, c_exp)
                                   : beam_search_team<FUSED, RK, 16>(v, s, scratch, cur, curd, efc, level, vc, c_dist, c_exp);
            }
            for (uint32_t i = ut; i < tsize; i += un) s.ti[i] &= kIdMask;
            sync();
            if (level == 0 && K > 0) {  // KNN-graph seed, hrnn.h:1479-1501
                uint32_t cnt = min(tsize, K);
                for (uint32_t i = ut; i < cnt; i += un) {
                    knn_ids[(size_t)p * K + i] = s.ti[i];
                    knn_dist[(size_t)p * K + i] = s.td[i];
                }
                if (ut == 0) knn_hdr[p] = cnt;
            }
            if (T > 1 && w != 0) continue;
            // (the visited cache is free here: it holds the kept rows)
            uint32_t ns = heuristic<FUSED, RK>(v, s.ti, s.td, tsize, M, (float*)s.vis, vc / v.dim, sel_id, sel_d,
                                               scratch);
            uint32_t* own = level == 0 ? adj0 + (size_t)p * v.W0 : upper + v.upper_off[p] + (size_t)(level - 1) * v.WU;
            for (uint32_t i = lane; i < ns; i += 32) own[1 + i] = sel_id[ns - 1 - i];  // farthest first
            if (lane == 0) own[0] = ns;
            // the links back
            uint32_t o0 = (p - b0) * M;  // this point's first number; above level 0 after all points'
            if (level > 0) {
                if (lane == 0) o0 = (b1 - b0) * M + atomicAdd(&lt.ctr[1], ns);
                o0 = __shfl_sync(0xFFFFFFFFu, o0, 0);
            }
            for (uint32_t i = lane; i < ns; i += 32) {
                const uint32_t t = sel_id[i], o = o0 + i;
                const uint32_t key = level == 0 ? t : cap + (uint32_t)(v.upper_off[t] / v.WU) + (uint32_t)(level - 1);
                const uint32_t at = atomicAdd(&lt.list[key].cnt, 1u), had = atomicCAS(&lt.list[key].rec, 0u, o + 1);
                const uint32_t rec = had ? had - 1 : o;
                const Link l{p, sel_d[i]};
                if (!had) lt.active[atomicAdd(&lt.ctr[0], 1u)] = ActiveList{key, t, rec};
                if (at < kSlots) lt.slot[(size_t)rec * kSlots + at] = l;
                else lt.over[o] = OverLink{l, atomicExch(&lt.head[rec], o)};
            }
            cur = sel_id[0];
            curd = sel_d[0];
            __syncwarp();
        }
        if constexpr (T > 1) __syncthreads();
    }
}

// Shared memory of one k_link_update warp.
__host__ __device__ inline size_t link_warp_bytes(uint32_t dim) {
    const size_t CMAX = kGroupMax + kMaxSel;
    return ((size_t)dim * 4 + CMAX * 8 + CMAX * 8 + kMaxSel * 12 + 64 * 4 + 15) & ~(size_t)15;
}

// One warp per target list with new links (mutuallyConnectNewElement, hrnn.h:729-797).
template <bool FUSED, int RK>
__global__ void __launch_bounds__(128, 4) k_link_update(DevView v, LinkTable lt, uint32_t cap, uint32_t maxM0,
                                                     uint32_t maxM, uint32_t* __restrict__ adj0,
                                                     uint32_t* __restrict__ upper) {
    extern __shared__ __align__(16) char smem_raw[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const uint32_t CMAX = kGroupMax + kMaxSel;
    char* base = smem_raw + (size_t)w * link_warp_bytes(v.dim);
    uint64_t* keys = (uint64_t*)base;                  // (d, id) sort keys; then the kept rows
    float* sq = (float*)(keys + CMAX);                 // target vector
    uint32_t* cid = (uint32_t*)(sq + v.dim);           // candidates, ascending
    float* cd = (float*)(cid + CMAX);
    uint32_t* sel_id = (uint32_t*)(cd + CMAX);
    float* sel_d = (float*)(sel_id + kMaxSel);
    uint32_t* eid = (uint32_t*)(sel_d + kMaxSel);      // existing links
    uint32_t* scratch = eid + kMaxSel;
    float* tmpd = (float*)scratch;
    const uint32_t na = lt.ctr[0];
    for (uint32_t g = blockIdx.x * wpb + w; g < na; g += gridDim.x * wpb) {
        const uint32_t key = lt.active[g].key, t = lt.active[g].target, rec = lt.active[g].rec;
        const uint32_t nn = min(lt.list[key].cnt, kGroupMax);
        const bool lvl0 = key < cap;
        uint32_t* list = lvl0 ? adj0 + (size_t)t * v.W0 : upper + (size_t)(key - cap) * v.WU;
        const uint32_t Mcur = lvl0 ? maxM0 : maxM;
        const uint32_t c0 = list[0] & 0xFFFFu;
        // new links sorted by (distance, id)
        uint32_t P = 32;
        while (P < nn) P <<= 1;
        for (uint32_t x = lane; x < P; x += 32) {
            uint64_t k = ~0ull;
            if (x < min(nn, kSlots)) {
                const Link l = lt.slot[(size_t)rec * kSlots + x];
                k = ((uint64_t)__float_as_uint(l.d) << 32) | l.src;
            }
            keys[x] = k;
        }
        if (nn > kSlots) {  // the overflow chain
            __syncwarp();
            if (lane == 0) {
                uint32_t o = lt.head[rec];
                for (uint32_t x = kSlots; x < nn; ++x) {
                    const OverLink e = lt.over[o];
                    keys[x] = ((uint64_t)__float_as_uint(e.l.d) << 32) | e.l.src;
                    o = e.next;
                }
                lt.head[rec] = kInvalid;
            }
        }
        __syncwarp();
        if (lane == 0) lt.list[key] = ListLinks{0u, 0u};  // ready for the next batch
        for (uint32_t kk = 2; kk <= P; kk <<= 1)
            for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
                __syncwarp();
                for (uint32_t x = lane; x < P; x += 32) {
                    uint32_t y = x ^ j;
                    if (y > x) {
                        uint64_t a = keys[x], c = keys[y];
                        if ((a > c) == ((x & kk) == 0)) {
                            keys[x] = c;
                            keys[y] = a;
                        }
                    }
                }
            }
        __syncwarp();
        if (c0 + nn <= Mcur) {  // room for all: append (hrnn.h:759-761)
            for (uint32_t x = lane; x < nn; x += 32) list[1 + c0 + x] = (uint32_t)keys[x];
            __syncwarp();
            if (lane == 0) list[0] = (list[0] & 0xFFFF0000u) | (c0 + nn);
            __syncwarp();
            continue;
        }
        // candidates: the new links and the existing ones with their distance to the
        // target (hrnn.h:766-774), then ordered by (distance, id)
        for (uint32_t e = lane; e < v.dim; e += 32) sq[e] = v.vec[(size_t)t * v.dim + e];
        for (uint32_t x = lane; x < c0; x += 32) eid[x] = list[1 + x];
        for (uint32_t x = lane; x < nn; x += 32) {
            cid[x] = (uint32_t)keys[x];
            cd[x] = __uint_as_float((uint32_t)(keys[x] >> 32));
        }
        __syncwarp();
        for (uint32_t bb = 0; bb < c0; bb += 32) {
            uint32_t cnt = min(32u, c0 - bb);
            warp_l2_list<FUSED, RK>(v, sq, eid + bb, cnt, tmpd);
            if ((uint32_t)lane < cnt) {
                cid[nn + bb + lane] = eid[bb + lane];
                cd[nn + bb + lane] = tmpd[lane];
            }
            __syncwarp();
        }
        const uint32_t total = c0 + nn;
        order_candidates(cid, cd, total, keys);
        for (uint32_t x = lane; x < total; x += 32) {
            cid[x] = (uint32_t)keys[x];
            cd[x] = __uint_as_float((uint32_t)(keys[x] >> 32));
        }
        __syncwarp();
        const uint32_t ns = heuristic<FUSED, RK>(v, cid, cd, total, Mcur, (float*)keys, CMAX * 2 / v.dim, sel_id, sel_d, scratch);
        for (uint32_t i = lane; i < ns; i += 32) list[1 + i] = sel_id[ns - 1 - i];
        __syncwarp();
        if (lane == 0) list[0] = (list[0] & 0xFFFF0000u) | ns;
        __syncwarp();
    }
}

int nsm_of(int dev) {
    int v = 148;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
}

}  // namespace

void add_points(Index& ix, const float* data, const uint64_t* labels, size_t n_add) {
    if (n_add == 0) return;
    if (ix.serve_mode) fail(HRNN_ERR_STATE, "addPoint: index is in serve mode");
    if (ix.cur + n_add > ix.max_elements)
        fail(HRNN_ERR_LIMIT, "The number of elements exceeds the specified limit");   // hrnn.h:1402-1404
    if (ix.maxM0 > kMaxSel || ix.M > kMaxSel) fail(HRNN_ERR_ARG, "addPoint: M above 32 is not supported");
    const size_t b_start = ix.cur, end = ix.cur + n_add, dim = ix.dim;
    std::vector<uint64_t> lab(n_add);
    for (size_t i = 0; i < n_add; ++i) {
        lab[i] = labels ? labels[i] : (uint64_t)(b_start + i);
        if (!ix.label_lookup.emplace(lab[i], (uint32_t)(b_start + i)).second) {
            for (size_t j = 0; j < i; ++j) ix.label_lookup.erase(lab[j]);
            fail(HRNN_ERR_ARG, "addPoint: label already present (updates are not supported)");
        }
    }
    cudaStream_t s = ix.stream;
    CUDA_CHECK(cudaMemcpyAsync(ix.vec.as<float>() + b_start * dim, data, n_add * dim * 4, cudaMemcpyHostToDevice, s));
    CUDA_CHECK(cudaMemcpyAsync(ix.labels.as<uint64_t>() + b_start, lab.data(), n_add * 8, cudaMemcpyHostToDevice, s));
    // Levels in insertion order from the reference's generator (hrnn.h:383-387).
    std::uniform_real_distribution<double> U(0.0, 1.0);
    for (size_t i = b_start; i < end; ++i) {
        int lv = (int)(-std::log(U(ix.level_generator)) * ix.mult);
        ix.levels[i] = lv;
        ix.upper_off[i] = ix.upper.size();
        if (lv > 0) ix.upper.resize(ix.upper.size() + (size_t)lv * (1 + ix.maxM), 0u);
    }
    ix.upper_dirty = true;
    ix.sync_upper_to_device();
    DevMem d_levels;
    d_levels.alloc(end * 4);
    CUDA_CHECK(cudaMemcpyAsync(d_levels.p, ix.levels.data(), end * 4, cudaMemcpyHostToDevice, s));
    // The batches: 1/24 of the index each, at most max_batch points.
    const size_t max_batch = 16384;
    size_t pos = b_start;
    if (ix.cur == 0 && ix.enterpoint == kInvalid) {  // first element (hrnn.h:1505-1509)
        ix.enterpoint = 0;
        ix.maxlevel = ix.levels[0];
        pos = 1;
    }
    struct Batch {
        size_t p0, p1;
        uint32_t ep;
        int maxlevel;
    };
    std::vector<Batch> batches;
    size_t maxreq = 1;  // the most links a batch can ask for: M on each of a point's levels
    for (; pos < end;) {
        const size_t p1 = std::min(end, pos + std::max<size_t>(1, std::min<size_t>(pos / 24, max_batch)));
        batches.push_back({pos, p1, ix.enterpoint, ix.maxlevel});
        size_t req = 0;
        for (size_t i = pos; i < p1; ++i) req += (size_t)(std::min(ix.levels[i], batches.back().maxlevel) + 1) * ix.M;
        maxreq = std::max(maxreq, req);
        // entry point: first point of the batch with the highest level above maxlevel
        for (size_t i = pos; i < p1; ++i)
            if (ix.levels[i] > ix.maxlevel) {
                ix.maxlevel = ix.levels[i];
                ix.enterpoint = (uint32_t)i;
            }
        pos = p1;
    }
    // The link table and the batches' counters (two each).
    const uint32_t cap = (uint32_t)ix.max_elements;
    const size_t keyspace = cap + ix.upper.size() / (1 + ix.maxM) + 1;
    DevMem klist, khead, kslot, kover, active, ctr;
    klist.alloc(keyspace * sizeof(ListLinks));
    khead.alloc(maxreq * 4);
    kslot.alloc(maxreq * kSlots * sizeof(Link));
    kover.alloc(maxreq * sizeof(OverLink));
    active.alloc(maxreq * sizeof(ActiveList));
    ctr.alloc(std::max<size_t>(batches.size(), 1) * 8);
    CUDA_CHECK(cudaMemsetAsync(klist.p, 0, klist.bytes, s));
    CUDA_CHECK(cudaMemsetAsync(khead.p, 0xFF, khead.bytes, s));
    CUDA_CHECK(cudaMemsetAsync(ctr.p, 0, ctr.bytes, s));
    LinkTable lt{klist.as<ListLinks>(), khead.as<uint32_t>(), kslot.as<Link>(), kover.as<OverLink>(),
                 active.as<ActiveList>(), nullptr};
    const int nsm = nsm_of(ix.device);
    const bool fused = (ix.order.fused & 1) != 0;
    const uint32_t efc = (uint32_t)((ix.ef_construction + 31) & ~(size_t)31);
    // Visited-cache slots per warp (lossy: a miss only re-scores a node, so the
    // graph does not depend on it); HRNN_BUILD_VC overrides, for measurements.
    uint32_t vc = 2048;
    if (const char* e = std::getenv("HRNN_BUILD_VC")) {
        const unsigned long v = std::strtoul(e, nullptr, 10);
        if (v >= 256 && v <= 8192 && (v & (v - 1)) == 0) vc = (uint32_t)v;
    }
    const size_t per_warp_b = build_warp_bytes((uint32_t)dim, efc, vc);
    const int wpb = (int)std::max<size_t>(1, std::min<size_t>(4, (200 * 1024) / per_warp_b));
    const size_t smem_b = per_warp_b * wpb;
    const size_t smem_l = link_warp_bytes((uint32_t)dim) * 4;
    if (smem_b > 227 * 1024 || smem_l > 227 * 1024) fail(HRNN_ERR_ARG, "addPoint: dim/ef_construction too large");
    const int rows = rows_kind((uint32_t)dim, ix.order.lanes);
    auto kb1 = with_rows(rows, [&](auto rk) {
        return fused ? k_build_batch<true, decltype(rk)::value, 1> : k_build_batch<false, decltype(rk)::value, 1>;
    });
    auto kbt = with_rows(rows, [&](auto rk) {
        constexpr int RK = decltype(rk)::value;
        if constexpr (RK == kRowsAny) return kb1;
        else return fused ? k_build_batch<true, RK, kTeamWarps> : k_build_batch<false, RK, kTeamWarps>;
    });
    // A team per point while a batch is too small to fill the device.
    const bool team_ok = rows != kRowsAny && efc <= kTeamMaxEf && ix.maxM0 <= 32 && ix.maxM <= 32 &&
                         build_warp_bytes((uint32_t)dim, efc, team_vis(efc)) <= 227 * 1024;
    const uint32_t team_vc = team_vis(efc);
    const size_t team_smem = build_warp_bytes((uint32_t)dim, efc, team_vc);
    const size_t team_points = team_searches(nsm);
    auto kl = with_rows(rows, [&](auto rk) {
        return fused ? k_link_update<true, decltype(rk)::value> : k_link_update<false, decltype(rk)::value>;
    });
    CUDA_CHECK(cudaFuncSetAttribute(kb1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_b));
    if (team_ok)
        CUDA_CHECK(cudaFuncSetAttribute(kbt, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)team_smem));
    CUDA_CHECK(cudaFuncSetAttribute(kl, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_l));
    // All batches are enqueued without waiting: a batch's sizes on the device
    // (active lists, links above level 0) are read there.
    for (size_t bi = 0; bi < batches.size(); ++bi) {
        const Batch& b = batches[bi];
        ix.cur = b.p1;  // view covers the batch (vectors); the graph does not reach it yet
        const DevView v = make_view(ix);
        lt.ctr = ctr.as<uint32_t>() + 2 * bi;
        const size_t nb = b.p1 - b.p0;
        const bool team = team_ok && nb <= team_points;
        // one warp per point: few points are spread over the SMs rather than packed
        const int cw = team ? kTeamWarps : (int)std::min<size_t>(wpb, (nb + nsm - 1) / nsm);
        const unsigned grid = (unsigned)std::min<size_t>(team ? nb : (nb + cw - 1) / cw, (size_t)nsm * 8);
        (team ? kbt : kb1)<<<grid, cw * 32, team ? team_smem : per_warp_b * cw, s>>>(
            v, (uint32_t)b.p0, (uint32_t)b.p1, b.ep, b.maxlevel, efc, team ? team_vc : vc, (uint32_t)ix.M, cap, d_levels.as<int32_t>(),
            (uint32_t)ix.K, ix.knn_hdr.as<uint32_t>(), ix.knn_ids.as<uint32_t>(), ix.knn_dist.as<float>(),
            ix.adj0.as<uint32_t>(), ix.d_upper.as<uint32_t>(), lt);
        CUDA_LAUNCH_CHECK();
        const unsigned gl = (unsigned)std::min<size_t>((nb * ix.M + 3) / 4, (size_t)nsm * 8);
        kl<<<std::max(1u, gl), 128, smem_l, s>>>(v, lt, cap, (uint32_t)ix.maxM0, (uint32_t)ix.maxM,
                                                 ix.adj0.as<uint32_t>(), ix.d_upper.as<uint32_t>());
        CUDA_LAUNCH_CHECK();
    }
    CUDA_CHECK(cudaStreamSynchronize(s));
    ix.cur = end;
    ix.bf16_valid = false;  // the BF16 / INT8 copies are rebuilt on the next search that uses them
    ix.i8_valid = false;
    // The reverse lists no longer cover every point: searches need buildRKNNG first
    // (the reference leaves its flag set and would read past its offsets array).
    ix.rknng_built = false;
    // The device copy of the upper layers is now authoritative; mirror it back.
    if (!ix.upper.empty())
        CUDA_CHECK(cudaMemcpy(ix.upper.data(), ix.d_upper.p, ix.upper.size() * 4, cudaMemcpyDeviceToHost));
    ix.upper_dirty = false;
}

}  // namespace hrnn
