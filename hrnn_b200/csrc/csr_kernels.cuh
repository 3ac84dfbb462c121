// Kernels that buildRKNNG (csr.cu) and its allocation-free form (csr_noalloc.cu)
// share: the scatter of a KNN graph's edges into their targets' segments and the
// sort of segments of up to kWarpSegMax entries.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace hrnn {
namespace {

constexpr int kEdgeU = 4;  // edges a lane of the scatter has on their way

// A transpose whose sizes the host does not wait for: nothing is written when the
// edges (*total, null: not asked) pass the entries' capacity or the graph is bad.
struct Guard {
    const uint64_t* total = nullptr;
    uint64_t cap = 0;
    const uint32_t* bad = nullptr;  // two counts
    __device__ __forceinline__ bool stop() const { return total && (*total > cap || bad[0] || bad[1]); }
};

// cursor[i]: where segment i's next entry goes, as an index into ent.  One atomic per
// edge gives its place: with the cursor counted from 0 and the segment's offset
// read beside it, a 200k x 100 graph's 20M edges took 330 us, bound by their random
// L2 accesses (three per edge; now two, 275 us).
template <class E, class C>
__global__ void k_scatter_edges(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ cnt, size_t n, uint32_t K,
                                C* __restrict__ cursor, E* __restrict__ ent, uint32_t rb, Guard guard) {
    if (guard.stop()) return;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const size_t nw = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t i = warp; i < n; i += nw) {
        const uint32_t c = cnt[i] & 0xFFFFu;
        const uint32_t* row = ids + i * K;
        for (uint32_t j0 = lane; j0 < c; j0 += 32 * kEdgeU) {
            uint32_t nbr[kEdgeU];
            C pos[kEdgeU];
#pragma unroll
            for (int u = 0; u < kEdgeU; ++u) nbr[u] = j0 + 32 * u < c ? row[j0 + 32 * u] : 0u;
#pragma unroll
            for (int u = 0; u < kEdgeU; ++u)
                if (j0 + 32 * u < c) pos[u] = atomicAdd(&cursor[nbr[u]], (C)1);
#pragma unroll
            for (int u = 0; u < kEdgeU; ++u)
                if (j0 + 32 * u < c) ent[pos[u]] = (E)(((uint64_t)i << rb) | (j0 + 32 * u));
        }
    }
}

// Sort keys: an entry with its rank bits rotated to the top, so keys order by (rank,
// owner) and are as wide as the entries.
__device__ __forceinline__ uint32_t seg_key(uint32_t e, uint32_t rb) { return __funnelshift_r(e, e, rb); }
__device__ __forceinline__ uint32_t seg_entry(uint32_t k, uint32_t rb) { return __funnelshift_l(k, k, rb); }
__device__ __forceinline__ uint64_t seg_key(uint64_t e, uint32_t rb) { return rb ? (e >> rb) | (e << (64 - rb)) : e; }
__device__ __forceinline__ uint64_t seg_entry(uint64_t k, uint32_t rb) { return rb ? (k << rb) | (k >> (64 - rb)) : k; }

// The warp's 32 R keys ascending, key lane * R + r in x[r]: a bitonic network whose
// merges start with the mirrored partner, so every comparison goes the same way;
// distances below R stay in a lane.
template <class T, int R>
__device__ __forceinline__ void warp_sort(T (&x)[R]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1) {
        // partner index ^ (k - 1)
        if (k <= R) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int q = r ^ (k - 1);
                if (r < q) {
                    const T a = x[r], b = x[q];
                    x[r] = a < b ? a : b;
                    x[q] = a < b ? b : a;
                }
            }
        } else {
            const bool low = (lane & (k / R / 2)) == 0;
            T y[R];
#pragma unroll
            for (int r = 0; r < R; ++r) y[r] = __shfl_xor_sync(0xFFFFFFFFu, x[R - 1 - r], k / R - 1);
#pragma unroll
            for (int r = 0; r < R; ++r) x[r] = (x[r] < y[r]) == low ? x[r] : y[r];
        }
        // partner index ^ j
#pragma unroll
        for (int j = k >> 2; j > 0; j >>= 1) {
            if (j >= R) {
                const bool low = (lane & (j / R)) == 0;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const T y = __shfl_xor_sync(0xFFFFFFFFu, x[r], j / R);
                    x[r] = (x[r] < y) == low ? x[r] : y;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if ((r & j) == 0) {
                        const T a = x[r], b = x[r | j];
                        x[r] = a < b ? a : b;
                        x[r | j] = a < b ? b : a;
                    }
            }
        }
    }
}

constexpr int kWarpSegMax = 1024;  // entries of a segment one warp sorts
constexpr int kSegWarps = 4;

template <class E, int R>
__device__ __forceinline__ void sort_segment(E* __restrict__ seg, uint32_t len, uint32_t rb, E* sm) {
    const int lane = threadIdx.x & 31;
    E x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = 32 * r + lane < len ? seg_key(seg[32 * r + lane], rb) : (E)~(E)0;
    warp_sort<E, R>(x);
#pragma unroll
    for (int r = 0; r < R; ++r) sm[lane * R + r] = x[r];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (32 * r + lane < len) seg[32 * r + lane] = seg_entry(sm[32 * r + lane], rb);
    __syncwarp();
}

// One warp per segment of up to kWarpSegMax entries, sorted in registers by (rank,
// owner); longer ones are listed in `big`, and the largest power of two at or above
// a listed length is kept in *max_p.  With 64-bit keys in shared memory the 200k
// segments of a 200k x 100 graph took 757 us, 32-bit keys in registers take 123 us.
template <class E>
__global__ void __launch_bounds__(32 * kSegWarps) k_sort_segments(const uint64_t* __restrict__ off, size_t n,
                                                                  E* __restrict__ ent, uint32_t rb,
                                                                  uint32_t* __restrict__ big,
                                                                  uint32_t* __restrict__ n_big,
                                                                  uint32_t* __restrict__ max_p, Guard guard) {
    if (guard.stop()) return;
    __shared__ E sm[kSegWarps][kWarpSegMax];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (size_t seg = (size_t)blockIdx.x * kSegWarps + w; seg < n; seg += (size_t)gridDim.x * kSegWarps) {
        const uint64_t b = off[seg], len = off[seg + 1] - b;
        if (len <= 1) continue;
        if (len > (uint64_t)kWarpSegMax) {
            if (lane == 0) {
                uint32_t P = 2 * kWarpSegMax;
                while (P < len) P <<= 1;
                big[atomicAdd(n_big, 1u)] = (uint32_t)seg;
                atomicMax(max_p, P);
            }
            continue;
        }
        const uint32_t m = (uint32_t)len;
        if (m <= 32) sort_segment<E, 1>(ent + b, m, rb, sm[w]);
        else if (m <= 64) sort_segment<E, 2>(ent + b, m, rb, sm[w]);
        else if (m <= 128) sort_segment<E, 4>(ent + b, m, rb, sm[w]);
        else if (m <= 256) sort_segment<E, 8>(ent + b, m, rb, sm[w]);
        else if (m <= 512) sort_segment<E, 16>(ent + b, m, rb, sm[w]);
        else sort_segment<E, 32>(ent + b, m, rb, sm[w]);
    }
}

}  // namespace
}  // namespace hrnn
