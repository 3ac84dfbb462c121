// Warp-level graph search shared by the query path (search.cu) and the batched
// HNSW construction (hnsw_build.cu): greedy descent over the upper layers and
// the best-first beam search of one layer, with the exact FP32 distance order.
//
// Beam formulation of searchBaseLayerST (hrnn.h:484-616): the result max-heap of
// size ef and the candidate min-heap are one ascending list in shared memory
// whose entries carry an "expanded" flag.  The next node to expand is the first
// unexpanded entry; neighbour j of an expansion is accepted iff fewer than ef
// elements of (beam before the expansion + earlier fresh neighbours) are <= d_j,
// which is the reference's sequential test (size < ef || bound > d_j) evaluated
// after the earlier neighbours (neighbours it rejected never change the count).
// The visited array is a lossy direct-mapped cache plus an exact membership test
// against the beam; a point evicted from the cache and met again is either in
// the beam (caught) or was rejected/popped before, in which case the acceptance
// test rejects it again.  Equal distances of different points are the only case
// in which the order can differ from the reference's heaps.
#pragma once

#include <cfloat>
#include <cstdlib>

#include "common.cuh"

namespace hrnn {

struct DevView {
    const float* vec;
    const uint32_t* adj0;
    const uint32_t* upper;
    const uint64_t* upper_off;
    const uint32_t* knn_hdr;
    const float* knn_dist;
    const float* kdist_serve;
    const uint64_t* csr_off;
    const void* csr_ent;
    const uint64_t* labels;
    const uint16_t* vec_bf16;  // mixed precision: BF16 rows (or null)
    const float* vec_err;      // ||x - bf16(x)||_2, rounded up
    const uint32_t* knn_ids;   // KNN slot ids (FP64 radius re-decision)
    const int8_t* vec_i8;      // INT8 beam: rows round(x / s) (or null)
    const float4* i8_meta;     // (s, ||x - s c||, sum c^2, 0) per row
    uint32_t n, dim, nb, W0, WU, K, mks, rank_bits;
    int maxlevel;
    uint32_t enterpoint;
    int wide, lanes, fused;
    int i8_screen;             // verification screens with the INT8 rows first
};

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    x ^= x >> 16;
    return x;
}

// Links of node c at `level`: word 0 = count (low 16 bits), then the ids.
__device__ __forceinline__ const uint32_t* links_of(const DevView& v, uint32_t c, int level) {
    if (level == 0) return v.adj0 + (size_t)c * v.W0;
    return v.upper + v.upper_off[c] + (size_t)(level - 1) * v.WU;
}

// One thread, one row, 16-lane order (the AVX-512 path of space_l2.h:25-54):
// accumulator l takes elements l, l+16, ...; the row is read with 16-byte loads,
// two 64-byte blocks at a time, so a warp keeps up to 32 rows in flight.  q is
// in shared memory (16-byte aligned); every thread reads the same q words.
template <bool FUSED>
__device__ __forceinline__ float l2_row16(const float* __restrict__ q, const float* __restrict__ x, uint32_t nb) {
    float acc[16];
#pragma unroll
    for (int l = 0; l < 16; ++l) acc[l] = 0.f;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const float4* q4 = reinterpret_cast<const float4*>(q);
    uint32_t i = 0;
    for (; i + 2 <= nb; i += 2) {
        float4 a[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) a[c] = __ldg(x4 + 4 * i + c);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float4 p = q4[4 * i + c];
            const int l = (c & 3) * 4;
            acc[l + 0] = sq_step(acc[l + 0], p.x - a[c].x, FUSED);
            acc[l + 1] = sq_step(acc[l + 1], p.y - a[c].y, FUSED);
            acc[l + 2] = sq_step(acc[l + 2], p.z - a[c].z, FUSED);
            acc[l + 3] = sq_step(acc[l + 3], p.w - a[c].w, FUSED);
        }
    }
    if (i < nb) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float4 a = __ldg(x4 + 4 * i + c);
            const float4 p = q4[4 * i + c];
            const int l = c * 4;
            acc[l + 0] = sq_step(acc[l + 0], p.x - a.x, FUSED);
            acc[l + 1] = sq_step(acc[l + 1], p.y - a.y, FUSED);
            acc[l + 2] = sq_step(acc[l + 2], p.z - a.z, FUSED);
            acc[l + 3] = sq_step(acc[l + 3], p.w - a.w, FUSED);
        }
    }
    float s = acc[0];
#pragma unroll
    for (int l = 1; l < 16; ++l) s = __fadd_rn(s, acc[l]);
    return s;
}

// Two lanes per row (lane parity p owns accumulators 8p..8p+7, i.e. float4 #2p and
// #2p+1 of every 16-element block); all of a lane's loads for its half row are
// issued before the accumulation, so 16 rows of a warp cost one memory round trip.
template <bool FUSED, int NB>
__device__ __forceinline__ float l2_pair16(const float* __restrict__ q, const float* __restrict__ x, int p) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const float4* q4 = reinterpret_cast<const float4*>(q);
    float4 a[2 * NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        a[2 * i] = __ldg(x4 + 4 * i + 2 * p);
        a[2 * i + 1] = __ldg(x4 + 4 * i + 2 * p + 1);
    }
    float acc[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) acc[l] = 0.f;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float4 qq = q4[4 * i + 2 * p + c];
            const float4 xx = a[2 * i + c];
            acc[4 * c + 0] = sq_step(acc[4 * c + 0], qq.x - xx.x, FUSED);
            acc[4 * c + 1] = sq_step(acc[4 * c + 1], qq.y - xx.y, FUSED);
            acc[4 * c + 2] = sq_step(acc[4 * c + 2], qq.z - xx.z, FUSED);
            acc[4 * c + 3] = sq_step(acc[4 * c + 3], qq.w - xx.w, FUSED);
        }
    }
    // TmpRes[0] + ... + TmpRes[15] left to right: the even lane owns 0..7.
    float hi[8];
#pragma unroll
    for (int l = 0; l < 8; ++l) hi[l] = __shfl_down_sync(0xFFFFFFFFu, acc[l], 1);
    float s = acc[0];
#pragma unroll
    for (int l = 1; l < 8; ++l) s = __fadd_rn(s, acc[l]);
#pragma unroll
    for (int l = 0; l < 8; ++l) s = __fadd_rn(s, hi[l]);
    return s;  // valid in the even lane
}

// Four lanes per row: lane c of the quad owns accumulators 4c .. 4c + 3, i.e. float4
// #c of every 16-element block, so a quad reads 64 contiguous bytes of its row and a
// load instruction of the warp touches 8 lines (two lanes per row: 16 lines, and
// the beam search was bound by L1 line lookups at 70-76 % of their peak).  The 16
// accumulators are summed left to right along the quad; the distance is valid in
// every lane of the quad.
__device__ __forceinline__ float quad_sum16(float a0, float a1, float a2, float a3) {
    const int lane = threadIdx.x & 31, c = lane & 3;
    float s = __fadd_rn(__fadd_rn(__fadd_rn(a0, a1), a2), a3);
#pragma unroll
    for (int k = 1; k < 4; ++k) {
        const float t = __shfl_sync(0xFFFFFFFFu, s, (lane & ~3) + k - 1);
        if (c == k) s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t, a0), a1), a2), a3);
    }
    return __shfl_sync(0xFFFFFFFFu, s, lane | 3);
}

// One 16-element block of a quad: lane c's four accumulators.
template <bool FUSED>
__device__ __forceinline__ void quad_step(float (&acc)[4], float4 q, float4 x) {
    acc[0] = sq_step(acc[0], q.x - x.x, FUSED);
    acc[1] = sq_step(acc[1], q.y - x.y, FUSED);
    acc[2] = sq_step(acc[2], q.z - x.z, FUSED);
    acc[3] = sq_step(acc[3], q.w - x.w, FUSED);
}

// Distances of q to vec rows ids[0..cnt), dim = 16 NB: eight rows at a time.
template <bool FUSED, int NB>
__device__ __forceinline__ void warp_l2_quads(const DevView& v, const float* q, const uint32_t* ids, uint32_t cnt,
                                              float* dout) {
    const int lane = threadIdx.x & 31, c = lane & 3, r = lane >> 2;
    const float4* q4 = reinterpret_cast<const float4*>(q) + c;
    for (uint32_t b = 0; b < cnt; b += 8) {
        float4 x[NB];
        const uint32_t t = b + r;
        const float4* x4 = reinterpret_cast<const float4*>(v.vec + (size_t)ids[t < cnt ? t : b] * (16 * NB)) + c;
#pragma unroll
        for (int i = 0; i < NB; ++i) x[i] = __ldg(x4 + 4 * i);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < NB; ++i) quad_step<FUSED>(acc, q4[4 * i], x[i]);
        const float d = quad_sum16(acc[0], acc[1], acc[2], acc[3]);
        if (c == 0 && t < cnt) dout[t] = d;
    }
}

// The same for any dim that is a multiple of 16, four blocks of two groups in flight.
template <bool FUSED>
__device__ __forceinline__ void warp_l2_quads_any(const DevView& v, const float* q, const uint32_t* ids, uint32_t cnt,
                                                  float* dout) {
    const int lane = threadIdx.x & 31, c = lane & 3, r = lane >> 2;
    const float4* q4 = reinterpret_cast<const float4*>(q) + c;
    for (uint32_t b = 0; b < cnt; b += 16) {
        const uint32_t t0 = b + r, t1 = b + 8 + r;
        const float4* x0 = reinterpret_cast<const float4*>(v.vec + (size_t)ids[t0 < cnt ? t0 : b] * v.dim) + c;
        const float4* x1 = reinterpret_cast<const float4*>(v.vec + (size_t)ids[t1 < cnt ? t1 : b] * v.dim) + c;
        float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t i = 0;
        for (; i + 4 <= v.nb; i += 4) {
            float4 u[4], w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                u[k] = __ldg(x0 + 4 * (i + k));
                w[k] = __ldg(x1 + 4 * (i + k));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float4 p = q4[4 * (i + k)];
                quad_step<FUSED>(a0, p, u[k]);
                quad_step<FUSED>(a1, p, w[k]);
            }
        }
        for (; i < v.nb; ++i) {
            const float4 p = q4[4 * i];
            quad_step<FUSED>(a0, p, __ldg(x0 + 4 * i));
            quad_step<FUSED>(a1, p, __ldg(x1 + 4 * i));
        }
        const float d0 = quad_sum16(a0[0], a0[1], a0[2], a0[3]), d1 = quad_sum16(a1[0], a1[1], a1[2], a1[3]);
        if (c == 0 && t0 < cnt) dout[t0] = d0;
        if (c == 0 && t1 < cnt) dout[t1] = d1;
    }
}

// dims that are a multiple of 4 but not of 16 (space_l2.h:214-238 takes the 4-lane
// order for all of them): lane l of the quad is accumulator l and reads elements l,
// l + 4, ..., sixteen bytes of the row per quad and load, kQ4 of two groups in flight.
template <bool FUSED>
__device__ __forceinline__ void warp_l2_quads4(const DevView& v, const float* q, const uint32_t* ids, uint32_t cnt,
                                               float* dout) {
    constexpr int kQ4 = 16;
    const int lane = threadIdx.x & 31, c = lane & 3, r = lane >> 2;
    const uint32_t n4 = v.dim >> 2;
    for (uint32_t b = 0; b < cnt; b += 16) {
        const uint32_t t0 = b + r, t1 = b + 8 + r;
        const float* x0 = v.vec + (size_t)ids[t0 < cnt ? t0 : b] * v.dim + c;
        const float* x1 = v.vec + (size_t)ids[t1 < cnt ? t1 : b] * v.dim + c;
        float a0 = 0.f, a1 = 0.f;
        for (uint32_t i = 0; i < n4; i += kQ4) {
            float u[kQ4], w[kQ4];
#pragma unroll
            for (int k = 0; k < kQ4; ++k)
                if (i + k < n4) {  // uniform
                    u[k] = __ldg(x0 + 4 * (i + k));
                    w[k] = __ldg(x1 + 4 * (i + k));
                }
#pragma unroll
            for (int k = 0; k < kQ4; ++k)
                if (i + k < n4) {
                    const float p = q[4 * (i + k) + c];
                    a0 = sq_step(a0, p - u[k], FUSED);
                    a1 = sq_step(a1, p - w[k], FUSED);
                }
        }
        float s0 = __shfl_sync(0xFFFFFFFFu, a0, 0, 4), s1 = __shfl_sync(0xFFFFFFFFu, a1, 0, 4);
#pragma unroll
        for (int k = 1; k < 4; ++k) {
            s0 = __fadd_rn(s0, __shfl_sync(0xFFFFFFFFu, a0, k, 4));
            s1 = __fadd_rn(s1, __shfl_sync(0xFFFFFFFFu, a1, k, 4));
        }
        if (c == 0 && t0 < cnt) dout[t0] = s0;
        if (c == 0 && t1 < cnt) dout[t1] = s1;
    }
}

// How the exact kernels read rows, a template parameter of theirs (with one kernel
// for all widths the widest path set the registers of every search): the width
// itself for the unrolled ones under the 16-lane order, kRows16 for its other
// multiples of 16, kRows4 for multiples of 4 that are no multiples of 16, kRowsAny
// for the rest and for the other orders' multiples of 16.
constexpr int kRows16 = 16, kRows4 = 4, kRowsAny = 0;

inline int rows_kind(uint32_t dim, int lanes) {
    if (dim % 16 == 0) {
        if (lanes != 16) return kRowsAny;
        return dim == 64 || dim == 96 || dim == 128 || dim == 256 ? (int)dim : kRows16;
    }
    return dim % 4 == 0 ? kRows4 : kRowsAny;
}

// Calls f with std::integral_constant<int, kind>.
template <class F>
auto with_rows(int kind, F&& f) {
    switch (kind) {
        case 64: return f(std::integral_constant<int, 64>{});
        case 96: return f(std::integral_constant<int, 96>{});
        case 128: return f(std::integral_constant<int, 128>{});
        case 256: return f(std::integral_constant<int, 256>{});
        case kRows16: return f(std::integral_constant<int, kRows16>{});
        case kRows4: return f(std::integral_constant<int, kRows4>{});
        default: return f(std::integral_constant<int, kRowsAny>{});
    }
}

// Distances of q to cnt (<= 32) stored vectors ids[0..cnt) -> dout[0..cnt).
template <bool FUSED, int RK>
__device__ __forceinline__ void warp_l2_list(const DevView& v, const float* q, const uint32_t* ids, uint32_t cnt,
                                             float* dout) {
    if constexpr (RK == kRows16) {
        warp_l2_quads_any<FUSED>(v, q, ids, cnt, dout);
    } else if constexpr (RK == kRows4) {
        warp_l2_quads4<FUSED>(v, q, ids, cnt, dout);
    } else if constexpr (RK == kRowsAny) {
        for (uint32_t t = threadIdx.x & 31; t < cnt; t += 32)
            dout[t] = l2_thread(q, v.vec + (size_t)ids[t] * v.dim, v.dim, v.lanes, v.fused);
    } else {
        warp_l2_quads<FUSED, RK / 16>(v, q, ids, cnt, dout);
    }
    __syncwarp();
}

struct WarpSmem {
    float* q;
    float* td;       // beam distances (ascending)
    uint32_t* ti;    // beam ids | kExpanded
    float* xd;       // merge scratch
    uint32_t* xi;
    uint32_t* vis;   // visited cache
    float* nd;       // neighbour distances
    uint32_t* ni;    // neighbour ids
    uint32_t* apos;  // accepted insertion points
    int* q8;         // INT8 beam: the query as packed int8 words (dim / 4)
    float4* qm;      // (s_q^2 sum q8^2, s_q, ||q - s_q q8||, 0)
};

__host__ __device__ inline size_t warp_smem_bytes(uint32_t dim, uint32_t efc, uint32_t vc) {
    // a multiple of 16 (efc is one of 32), like every part's place
    return (((size_t)dim * 4 + 15) & ~(size_t)15) + (((size_t)dim + 15) & ~(size_t)15) + 16 + (size_t)(efc + 32) * 8 + (size_t)vc * 4 +
           32 * 12 + 16;
}

// q | q8 (dim bytes, padded to 16) | qm (16 bytes) | td | ti | vis | nd | ni | apos
__device__ inline WarpSmem carve(char* base, uint32_t dim, uint32_t efc, uint32_t vc) {
    WarpSmem s;
    s.q = (float*)base;
    base += ((size_t)dim * 4 + 15) & ~(size_t)15;
    s.q8 = (int*)base;
    base += ((size_t)dim + 15) & ~(size_t)15;
    s.qm = (float4*)base;
    base += 16;
    s.td = (float*)base;
    base += (size_t)(efc + 32) * 4;
    s.ti = (uint32_t*)base;
    base += (size_t)(efc + 32) * 4;
    s.xd = nullptr;
    s.xi = nullptr;
    s.vis = (uint32_t*)base;
    base += (size_t)vc * 4;
    s.nd = (float*)base;
    base += 32 * 4;
    s.ni = (uint32_t*)base;
    base += 32 * 4;
    s.apos = (uint32_t*)base;
    return s;
}

// The INT8 query words and scalars that follow a warp's q (carve's layout).
__device__ __forceinline__ const int* i8_q_words(const float* q, uint32_t dim) {
    return reinterpret_cast<const int*>(q + dim);
}
__device__ __forceinline__ const float4* i8_q_meta(const float* q, uint32_t dim) {
    return reinterpret_cast<const float4*>(reinterpret_cast<const char*>(q + dim) + ((dim + 15) & ~15u));
}

// Words of the link row of c at `level`, loaded unconditionally (no dependence on
// the count): lane j gets word j (j < row width), lane 0 also word 32 (rows of 33
// words, maxM0 = 32).  All loads stay inside the row.
__device__ __forceinline__ void load_row(const DevView& v, uint32_t c, int level, uint32_t& w0, uint32_t& w1) {
    const int lane = threadIdx.x & 31;
    const uint32_t W = level == 0 ? v.W0 : v.WU;
    const uint32_t* row = links_of(v, c, level);
    w0 = (uint32_t)lane < W ? __ldg(row + lane) : 0u;
    w1 = (lane == 0 && W > 32) ? __ldg(row + 32) : 0u;
}

// ---------------------------------------------------------------------------
// BF16 rows (mixed-precision search): vec_bf16[n][dim] holds round-to-nearest
// copies of the FP32 rows.  These distances rank candidates only; every
// accept/reject decision is re-made against the FP32 rows (search_bc.cu).
// ---------------------------------------------------------------------------

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Two lanes per row, NB 16-element blocks: lane parity p reads bytes
// [64p, 64p+64) of every 128-byte chunk, i.e. elements 32c + 16p .. 32c + 16p + 15
// of chunk c; accumulation order is free (FP32, fused).
template <int NB>
struct Bf16Half {  // a lane's half of a row
    uint4 a[NB];
    __device__ __forceinline__ void load(const uint16_t* __restrict__ x, int p) {
        const uint4* x4 = reinterpret_cast<const uint4*>(x);
#pragma unroll
        for (int c = 0; c < NB / 2; ++c) {
            a[2 * c] = __ldg(x4 + 4 * c + 2 * p);
            a[2 * c + 1] = __ldg(x4 + 4 * c + 2 * p + 1);
        }
    }
    __device__ __forceinline__ float dist(const float* __restrict__ q, int p) const {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int c = 0; c < NB / 2; ++c) {  // 32-element chunks
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 w = a[2 * c + h];
                const float* qq = q + 32 * c + 16 * p + 8 * h;
                float t;
                t = qq[0] - bf16_lo(w.x); s0 = fmaf(t, t, s0);
                t = qq[1] - bf16_hi(w.x); s1 = fmaf(t, t, s1);
                t = qq[2] - bf16_lo(w.y); s0 = fmaf(t, t, s0);
                t = qq[3] - bf16_hi(w.y); s1 = fmaf(t, t, s1);
                t = qq[4] - bf16_lo(w.z); s0 = fmaf(t, t, s0);
                t = qq[5] - bf16_hi(w.z); s1 = fmaf(t, t, s1);
                t = qq[6] - bf16_lo(w.w); s0 = fmaf(t, t, s0);
                t = qq[7] - bf16_hi(w.w); s1 = fmaf(t, t, s1);
            }
        }
        const float s = s0 + s1;
        return s + __shfl_xor_sync(0xFFFFFFFFu, s, 1);  // both lanes of the pair
    }
};

template <int NB>
__device__ __forceinline__ float bf16_pair(const float* __restrict__ q, const uint16_t* __restrict__ x, int p) {
    Bf16Half<NB> h;
    h.load(x, p);
    return h.dist(q, p);
}

// Any dim (one lane per row, scalar), for dims not a multiple of 32.
__device__ __forceinline__ float bf16_thread(const float* __restrict__ q, const uint16_t* __restrict__ x, uint32_t d) {
    float s = 0.f;
    for (uint32_t e = 0; e < d; ++e) {
        float t = q[e] - __uint_as_float((uint32_t)x[e] << 16);
        s = fmaf(t, t, s);
    }
    return s;
}

// ---------------------------------------------------------------------------
// INT8 rows (INT8 beam): x ~ s c, c in [-127, 127]; the query is quantised the
// same way (s_q, q8) by the warp that searches it.  The approximate squared
// distance ||s_q q8 - s c||^2 = s_q^2 sum q8^2 + s^2 sum c^2 - 2 s_q s (q8 . c)
// takes integer dot products (dp4a) only; it ranks the beam, nothing else.
// ---------------------------------------------------------------------------

// The warp quantises s.q (FP32, dim floats) into s.q8 / s.qm.
__device__ __forceinline__ void i8_prep_query(const WarpSmem& s, uint32_t dim) {
    const int lane = threadIdx.x & 31;
    float mx = 0.f;
    for (uint32_t j = lane; j < dim; j += 32) mx = fmaxf(mx, fabsf(s.q[j]));
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    const float sc = mx > 0.f ? mx / 127.f : 1.f;
    int8_t* q8b = reinterpret_cast<int8_t*>(s.q8);
    double e2 = 0.0;
    int c2 = 0;
    for (uint32_t j = lane; j < dim; j += 32) {
        const int c = max(-127, min(127, __float2int_rn(s.q[j] / sc)));
        q8b[j] = (int8_t)c;
        const double dlt = (double)s.q[j] - (double)sc * (double)c;
        e2 += dlt * dlt;
        c2 += c * c;
    }
    for (int o = 16; o; o >>= 1) {
        e2 += __shfl_xor_sync(0xFFFFFFFFu, e2, o);
        c2 += __shfl_xor_sync(0xFFFFFFFFu, c2, o);
    }
    if (lane == 0) *s.qm = make_float4(sc * sc * (float)c2, sc, __double2float_ru(sqrt(e2)), 0.f);
    __syncwarp();
}

// NW 16-byte words of one row (dim = 16 NW), all loaded before the dot products.
template <int NW>
__device__ __forceinline__ float i8_row(const int* __restrict__ q8, float4 qm, const int8_t* __restrict__ x,
                                        float4 xm) {
    const int4* x4 = reinterpret_cast<const int4*>(x);
    int4 a[NW];
#pragma unroll
    for (int c = 0; c < NW; ++c) a[c] = __ldg(x4 + c);
    int dot = 0;
#pragma unroll
    for (int c = 0; c < NW; ++c) {
        dot = __dp4a(a[c].x, q8[4 * c + 0], dot);
        dot = __dp4a(a[c].y, q8[4 * c + 1], dot);
        dot = __dp4a(a[c].z, q8[4 * c + 2], dot);
        dot = __dp4a(a[c].w, q8[4 * c + 3], dot);
    }
    return qm.x + xm.x * xm.x * xm.z - 2.f * qm.y * xm.x * (float)dot;
}

template <int NW>
__device__ __forceinline__ void warp_i8_rows(const DevView& v, const int* q8, float4 qm, const uint32_t* ids,
                                             uint32_t cnt, float* dout) {
    const int lane = threadIdx.x & 31;
    for (uint32_t r = 0; r < cnt; r += 32) {
        const uint32_t t = r + lane;
        const uint32_t id = ids[t < cnt ? t : r];
        const float d = i8_row<NW>(q8, qm, v.vec_i8 + (size_t)id * v.dim, __ldg(v.i8_meta + id));
        if (t < cnt) dout[t] = d;
    }
}

__device__ __forceinline__ void warp_i8_list(const DevView& v, const int* q8, float4 qm, const uint32_t* ids,
                                             uint32_t cnt, float* dout) {
    // dim = 16 NW exactly (the precision setter allows multiples of 16 up to 256)
    switch (v.dim >> 4) {
#define HRNN_I8_CASE(W) \
    case W: warp_i8_rows<W>(v, q8, qm, ids, cnt, dout); break;
        HRNN_I8_CASE(1) HRNN_I8_CASE(2) HRNN_I8_CASE(3) HRNN_I8_CASE(4) HRNN_I8_CASE(5) HRNN_I8_CASE(6)
        HRNN_I8_CASE(7) HRNN_I8_CASE(8) HRNN_I8_CASE(9) HRNN_I8_CASE(10) HRNN_I8_CASE(11) HRNN_I8_CASE(12)
        HRNN_I8_CASE(13) HRNN_I8_CASE(14) HRNN_I8_CASE(15) HRNN_I8_CASE(16)
#undef HRNN_I8_CASE
        default: break;
    }
    __syncwarp();
}

// Cooperative INT8 row reads.  In round i of a block of eight rounds, lane
// (g, s) = (lane >> 3, lane & 7) reads bytes 16 s .. 16 s + 15 of row 4 i + g of a
// block of 32 rows, so one 16-byte load per lane covers four whole rows (one
// 128-byte line each) instead of 32 scattered ones; lanes with s >= NB (rows
// narrower than 128 bytes) read nothing.
template <int NB>
__device__ __forceinline__ int4 coop_i8_load(const int8_t* vec, uint32_t id) {
    const int s = threadIdx.x & 7;
    return s < NB ? __ldg(reinterpret_cast<const int4*>(vec + (size_t)id * (NB * 16)) + s) : make_int4(0, 0, 0, 0);
}

__device__ __forceinline__ int dp4a4(int4 a, int4 b) {
    return __dp4a(a.x, b.x, __dp4a(a.y, b.y, __dp4a(a.z, b.z, __dp4a(a.w, b.w, 0))));
}

// The row of a block whose whole dot product coop_sum8 leaves in this lane.
__device__ __forceinline__ uint32_t coop_row() { return 4 * (threadIdx.x & 7) + ((threadIdx.x >> 3) & 3); }

// Folds the eight partial dot products p[i] (round i) of the lanes of a group of
// eight so that lane (g, s) ends with the sum over the group of p[s] -- the whole
// dot product of row 4 s + g.  Three butterfly steps, each swapping half of the
// values still held: 4 + 2 + 1 shuffles for eight rows.
__device__ __forceinline__ int coop_sum8(const int (&p)[8]) {
    const int s = threadIdx.x & 7;
    const bool b2 = s & 4, b1 = s & 2, b0 = s & 1;
    int w[4], x[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int send = b2 ? p[k] : p[k + 4], keep = b2 ? p[k + 4] : p[k];
        w[k] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 4);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int send = b1 ? w[k] : w[k + 2], keep = b1 ? w[k + 2] : w[k];
        x[k] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 2);
    }
    const int send = b0 ? x[0] : x[1], keep = b0 ? x[1] : x[0];
    return keep + __shfl_xor_sync(0xFFFFFFFFu, send, 1);
}

// This lane's INT8 query words for the cooperative reads (bytes 16 s .. 16 s + 15).
template <int NB>
__device__ __forceinline__ int4 coop_q_words(const int* q8) {
    const int s = threadIdx.x & 7;
    return s < NB ? make_int4(q8[4 * s], q8[4 * s + 1], q8[4 * s + 2], q8[4 * s + 3]) : make_int4(0, 0, 0, 0);
}

// One row scored by every lane (the entry point of a search).
__device__ __forceinline__ float i8_one(const DevView& v, const float* q, uint32_t id) {
    const int* q8 = i8_q_words(q, v.dim);
    const float4 qm = *i8_q_meta(q, v.dim);
    const int8_t* x = v.vec_i8 + (size_t)id * v.dim;
    const float4 xm = __ldg(v.i8_meta + id);
    switch (v.dim >> 4) {
#define HRNN_I8_ONE(W) \
    case W: return i8_row<W>(q8, qm, x, xm);
        HRNN_I8_ONE(1) HRNN_I8_ONE(2) HRNN_I8_ONE(3) HRNN_I8_ONE(4) HRNN_I8_ONE(5) HRNN_I8_ONE(6)
        HRNN_I8_ONE(7) HRNN_I8_ONE(8) HRNN_I8_ONE(9) HRNN_I8_ONE(10) HRNN_I8_ONE(11) HRNN_I8_ONE(12)
        HRNN_I8_ONE(13) HRNN_I8_ONE(14) HRNN_I8_ONE(15) HRNN_I8_ONE(16)
#undef HRNN_I8_ONE
        default: return 0.f;
    }
}

// G: groups of 16 rows in flight.
template <int NB, int G = 1>
__device__ __forceinline__ void warp_bf16_pairs(const DevView& v, const float* q, const uint32_t* ids, uint32_t cnt,
                                                float* dout) {
    const int lane = threadIdx.x & 31, p = lane & 1;
    for (uint32_t r = 0; r < cnt; r += 16 * G) {
        Bf16Half<NB> h[G];
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (g == 0 || r + 16 * g < cnt) {  // uniform over the warp
                const uint32_t t = r + 16 * g + (lane >> 1);
                h[g].load(v.vec_bf16 + (size_t)ids[t < cnt ? t : r] * (16 * NB), p);
            }
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (g == 0 || r + 16 * g < cnt) {
                const uint32_t t = r + 16 * g + (lane >> 1);
                const float d = h[g].dist(q, p);
                if (p == 0 && t < cnt) dout[t] = d;
            }
    }
}

// Distance modes: 0 = exact FP32 unfused, 1 = exact FP32 fused, 2 = BF16 rows.
template <int DM, int RK = kRowsAny>
__device__ __forceinline__ void warp_dist_list(const DevView& v, const float* q, const uint32_t* ids, uint32_t cnt,
                                               float* dout) {
    if constexpr (DM == 3 && RK >= 64) {
        // q is the warp's s.q; its INT8 copy and (s_q^2 sum q8^2, s_q, e_q) follow it
        warp_i8_rows<RK / 16>(v, i8_q_words(q, RK), *i8_q_meta(q, RK), ids, cnt, dout);
        __syncwarp();
    } else if constexpr (DM == 3) {
        warp_i8_list(v, i8_q_words(q, v.dim), *i8_q_meta(q, v.dim), ids, cnt, dout);
    } else if constexpr (DM < 2) {
        warp_l2_list<DM == 1, RK>(v, q, ids, cnt, dout);
    } else {
        const int lane = threadIdx.x & 31;
        if constexpr (RK >= 64) {
            warp_bf16_pairs<RK / 16>(v, q, ids, cnt, dout);
        } else {
            for (uint32_t t = lane; t < cnt; t += 32) dout[t] = bf16_thread(q, v.vec_bf16 + (size_t)ids[t] * v.dim, v.dim);
        }
        __syncwarp();
    }
}

template <int DM, int RK = kRowsAny>
__device__ __forceinline__ float warp_dist_one(const DevView& v, const float* q, uint32_t id) {
    if constexpr (DM < 2 && RK != kRowsAny && RK != kRows4) {
        return l2_half16<DM == 1>(q, v.vec + (size_t)id * v.dim, v.nb, threadIdx.x & 15);
    } else if constexpr (DM < 2) {
        return l2_thread(q, v.vec + (size_t)id * v.dim, v.dim, v.lanes, v.fused);
    } else if constexpr (DM == 3 && RK >= 64) {
        return i8_row<RK / 16>(i8_q_words(q, RK), *i8_q_meta(q, RK), v.vec_i8 + (size_t)id * RK, __ldg(v.i8_meta + id));
    } else if constexpr (DM == 3) {
        return i8_one(v, q, id);
    } else {
        return bf16_thread(q, v.vec_bf16 + (size_t)id * v.dim, v.dim);
    }
}

// Greedy descent over levels top..stop+1 (hrnn.h:1992-2013, 1438-1464): per level,
// move to the first strict improvement of the running minimum in list order
// until a whole list brings none.  cur/curd are updated in every lane.
template <int DM, int RK>
__device__ void greedy_descent(const DevView& v, WarpSmem& s, int top, int stop, uint32_t& cur, float& curd,
                               unsigned long long& c_dist) {
    const int lane = threadIdx.x & 31;
    for (int level = top; level > stop; --level) {
        bool changed = true;
        while (changed) {
            changed = false;
            const uint32_t* blk = links_of(v, cur, level);
            const uint32_t w0 = (uint32_t)lane < v.WU ? blk[lane] : 0u;  // the row's first words in one load
            const uint32_t size = __shfl_sync(0xFFFFFFFFu, w0, 0) & 0xFFFFu;
            const uint32_t first = __shfl_sync(0xFFFFFFFFu, w0, (lane + 1) & 31);
            float bestd = curd;
            uint32_t best = cur;
            for (uint32_t base = 0; base < size; base += 32) {
                uint32_t cnt = min(32u, size - base);
                if ((uint32_t)lane < cnt) s.ni[lane] = base == 0 && lane < 31 ? first : blk[1 + base + lane];
                __syncwarp();
                warp_dist_list<DM, RK>(v, s.q, s.ni, cnt, s.nd);
                c_dist += cnt;
                // (idle lanes: no improvement even where the distances so far are infinite)
                float d = (uint32_t)lane < cnt ? s.nd[lane] : __uint_as_float(0x7F800000u);
                float mn = d;
                for (int o = 16; o; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
                uint32_t hit = __ballot_sync(0xFFFFFFFFu, (uint32_t)lane < cnt && d == mn);
                if (mn < bestd) {
                    bestd = mn;
                    best = s.ni[__ffs(hit) - 1];
                    changed = true;
                }
                __syncwarp();
            }
            cur = best;
            curd = bestd;
        }
    }
}

// keys[0..n) = the n candidates (distinct ids) by (distance, id): distance bits << 32 |
// id.  The distances are >= 0 or NaN, so their bits order as they do and a NaN has a
// place of its own, last.
__device__ __forceinline__ void order_candidates(const uint32_t* id, const float* d, uint32_t n, uint64_t* keys) {
    for (uint32_t x = threadIdx.x & 31; x < n; x += 32) {
        const uint32_t dx = __float_as_uint(d[x]), ix = id[x];
        uint32_t r = 0;
        for (uint32_t y = 0; y < n; ++y) {
            const uint32_t dy = __float_as_uint(d[y]);
            r += (dy < dx) || (dy == dx && id[y] < ix);
        }
        keys[r] = ((uint64_t)dx << 32) | ix;
    }
    __syncwarp();
}

// Number of td[0..n) that are not above x (the insertion point after equal
// distances; x is no NaN, which are above everything), for the lanes that ask: a
// search with three probes a round, four rounds for 200 entries instead of eight
// dependent shared-memory reads.
__device__ __forceinline__ uint32_t insert_pos(const float* td, uint32_t n, float x) {
    uint32_t step = 1, pos = 0;
    while (step * 4 <= n) step *= 4;  // uniform: n is the warp's
    for (; step; step >>= 2) {
        const uint32_t i0 = pos + step - 1, i1 = i0 + step, i2 = i1 + step;
        const float t0 = td[min(i0, n - 1)], t1 = td[min(i1, n - 1)], t2 = td[min(i2, n - 1)];
        const uint32_t c = (uint32_t)(i0 < n && t0 <= x) + (uint32_t)(i1 < n && t1 <= x) +
                           (uint32_t)(i2 < n && t2 <= x);
        pos += c * step;
    }
    return pos;
}

// A whole number that orders as the distance does (the INT8 form's may come out below
// 0), NaN last.
__device__ __forceinline__ int order_key(float d) {
    const int b = (int)__float_as_uint(d);
    return b ^ (b >> 31 & 0x7FFFFFFF);
}

// Inserts the scored neighbours of the lanes with `have` (d, id) into the beam:
// neighbour j is accepted iff fewer than EF elements of (beam + accepted earlier neighbours of
// this batch) are <= d_j, and not already in the beam; the beam stays sorted and
// is cut to EF; cursor moves back to the first inserted position.
//
// A neighbour no closer than the last entry of a full beam can be dropped before
// the rest: it would land at position EF, and it only counts against neighbours
// that are no closer than itself.  The others are all placed by (distance, beam
// entries first, lane): one that the sequential test rejects has at least EF
// elements before it in that order, so it falls beyond the cut, and so does
// whatever it would have moved.
//
// The beam is shifted 128 entries (four per lane) at a time from the right, each
// entry by the number of insertion points at or before it: counting them costs less
// than a search per entry, and the four entries' reads, counts and writes overlap.  (One 32-entry block at a time with a
// binary search per entry, and shuffle loops for both rankings, took about two
// thirds of the 8,000 cycles an expansion of a lone query cost at ef = 200.)
//
// A NaN distance (a NaN in the query or the row) is farther than every number and as
// far as another NaN, the order of the bits that the team search compares: it goes to
// the end of the beam and never enters a full one.
//
// known(d, ok, id, pos) is called by the whole warp once the neighbours to insert are
// known (lanes with ok), before the beam changes.  DEDUP: an id may come twice (two
// parents sharing a neighbour that the lossy visited cache did not catch): the lowest
// lane keeps it.
template <bool DEDUP = false, class F>
__device__ __forceinline__ void beam_insert(WarpSmem& s, float d, uint32_t id, bool have, uint32_t EF, uint32_t& tsize,
                                            uint32_t& cursor, F&& known) {
    const int lane = threadIdx.x & 31;
    const bool nan = d != d;
    bool ok = have && !(tsize >= EF && (nan || d >= s.td[EF - 1]));
    uint32_t pos = 0, ab = __ballot_sync(0xFFFFFFFFu, ok);
    if (ab) {
        if constexpr (DEDUP) {
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, ok ? id : kInvalid);
            if (ok && (same & lanemask_lt() & ab)) ok = false;
        }
        pos = insert_pos(s.td, tsize, d);
        if (nan) pos = tsize;
        if (ok) {
            for (int k = (int)pos - 1; k >= 0 && __float_as_uint(s.td[k]) == __float_as_uint(d); --k)
                if (((s.ti[k] ^ id) & kIdMask) == 0) {
                    ok = false;
                    break;
                }
        }
        ab = __ballot_sync(0xFFFFFFFFu, ok);
    }
    known(d, ok, id, pos);
    if (!ab) return;
    const uint32_t na = __popc(ab), me = __popc(ab & lanemask_lt());
    // ranks among the accepted ones, then their insertion points in that order, four
    // at a time from shared memory (s.nd has been read: the callers hold d in registers)
    const bool pad = (uint32_t)lane >= na && (uint32_t)lane < ((na + 3) & ~3u);
    const int key = order_key(d);
    int* const nk = reinterpret_cast<int*>(s.nd);
    if (ok) nk[me] = key;
    if (pad) nk[lane] = 0x7FFFFFFF;
    __syncwarp();
    uint32_t before = 0;
    for (uint32_t i = 0; i < na; i += 4) {
        const int4 o = *reinterpret_cast<const int4*>(nk + i);
        before += (uint32_t)(o.x < key || (o.x == key && i < me)) + (uint32_t)(o.y < key || (o.y == key && i + 1 < me)) +
                  (uint32_t)(o.z < key || (o.z == key && i + 2 < me)) + (uint32_t)(o.w < key || (o.w == key && i + 3 < me));
    }
    if (ok) s.apos[before] = pos;
    if (pad) s.apos[lane] = 0xFFFFFFFFu;
    __syncwarp();
    const uint32_t lo = s.apos[0];
    const uint32_t newsize = min(tsize + na, EF);
    // every chunk is read before any lane writes, and its targets lie in itself or
    // in chunks to its right that were already moved
    if (tsize > lo) {
        for (int b = (int)lo + (int)(((tsize - lo - 1) / 128) * 128); b >= (int)lo; b -= 128) {
            float dk[4];
            uint32_t ik[4], np[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t k = (uint32_t)b + 32 * u + lane;
                dk[u] = k < tsize ? s.td[k] : 0.f;
                ik[u] = k < tsize ? s.ti[k] : 0u;
                np[u] = k < tsize ? k : 0xFFFF0000u;
            }
            for (uint32_t i = 0; i < na; i += 4) {
                const uint4 p = *reinterpret_cast<const uint4*>(s.apos + i);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t k = (uint32_t)b + 32 * u + lane;
                    np[u] += (uint32_t)(p.x <= k) + (uint32_t)(p.y <= k) + (uint32_t)(p.z <= k) + (uint32_t)(p.w <= k);
                }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (np[u] < newsize) {
                    s.td[np[u]] = dk[u];
                    s.ti[np[u]] = ik[u];
                }
            __syncwarp();
        }
    }
    const uint32_t npos = pos + before;
    if (ok && npos < newsize) {
        s.td[npos] = d;
        s.ti[npos] = id;
    }
    tsize = newsize;
    cursor = min(cursor, lo);
    __syncwarp();
}

// The first unexpanded beam entry at or after position b and its position
// (kInvalid: none), in every lane.
__device__ __forceinline__ uint32_t first_unexpanded(const WarpSmem& s, uint32_t b, uint32_t tsize, uint32_t& at) {
    const int lane = threadIdx.x & 31;
    for (; b < tsize; b += 32) {
        const uint32_t idx = b + lane;
        const uint32_t t = idx < tsize ? s.ti[idx] : kExpanded;
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, !(t & kExpanded));
        if (bal) {
            at = b + __ffs(bal) - 1;
            return __shfl_sync(0xFFFFFFFFu, t, __ffs(bal) - 1);
        }
    }
    return kInvalid;
}

// The entry a best-first search expands next and the position it will have, given
// the neighbours of the one just expanded that are about to be inserted (lanes with
// ok: distance d, insertion point pos) and the unexpanded beam entry after it
// (`after` at `at`; kInvalid: none): the closest of them, the beam's at equal
// distance.  None of the inserted ones then lands before it, and it lands in the beam:
// in a full one the neighbours with ok are closer than the last entry.
__device__ __forceinline__ uint32_t next_entry(const WarpSmem& s, float d, bool ok, uint32_t id, uint32_t pos,
                                               uint32_t after, uint32_t& at) {
    // distances are >= 0 or NaN: their bits order as they do, NaN last
    const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, ok ? __float_as_uint(d) : 0xFFFFFFFFu);
    const uint32_t have = __ballot_sync(0xFFFFFFFFu, ok && __float_as_uint(d) == best);
    if (!have || (after != kInvalid && best >= __float_as_uint(s.td[at]))) return after;
    const int i = __ffs(have) - 1;
    at = __shfl_sync(0xFFFFFFFFu, pos, i);
    return __shfl_sync(0xFFFFFFFFu, id, i);
}

// Best-first search of one layer from (ep, epd) with beam size EF (<= efc).
// On return the beam s.td/s.ti[0..tsize) holds the EF nearest found, ascending
// (ids still carry the expanded flag).  vc: visited-cache slots (power of two).
template <int DM, int RK>
__device__ uint32_t beam_search(const DevView& v, WarpSmem& s, uint32_t ep, float epd, uint32_t EF, int level,
                                uint32_t vc, unsigned long long& c_dist, unsigned long long& c_exp) {
    const int lane = threadIdx.x & 31;
    for (uint32_t i = lane; i < vc; i += 32) s.vis[i] = kInvalid;
    __syncwarp();
    // Rows of at most 33 words (maxM0 <= 32) are read whole by the warp in one go.
    const bool short_rows = (level == 0 ? v.W0 : v.WU) <= 33;
    uint32_t tsize = 1, cursor = 0;
    if (lane == 0) {
        s.td[0] = epd;
        s.ti[0] = ep;
        s.vis[hash32(ep) & (vc - 1)] = ep;
    }
    __syncwarp();
    // The entry to expand (c, at position found), its link row on its way: known and
    // loaded before the beam is updated with the neighbours of the one before it
    // (next_entry) where a link row is a single load, else found by a scan.
    uint32_t c = ep, found = 0, row0 = 0, row1 = 0;
    if (short_rows) load_row(v, c, level, row0, row1);
    // (no node is expanded twice, so v.n steps always do)
    uint32_t steps = 0;
    while (c != kInvalid && steps < v.n) {
        if (lane == 0) s.ti[found] = c | kExpanded;
        cursor = found + 1;
        uint32_t at = 0, after = kInvalid;
        if (short_rows) after = first_unexpanded(s, cursor, tsize, at);
        steps++;
        const uint32_t* adj = links_of(v, c, level);
        if (!short_rows) row0 = adj[0];
        const uint32_t size = __shfl_sync(0xFFFFFFFFu, row0, 0) & 0xFFFFu;
        bool known = false;
        for (uint32_t base = 0; base < size; base += 32) {
            uint32_t j = base + lane;
            uint32_t nid;
            if (short_rows) {  // id j is word j + 1 of the row
                const uint32_t a = __shfl_sync(0xFFFFFFFFu, row0, (lane + 1) & 31);
                const uint32_t b = __shfl_sync(0xFFFFFFFFu, row1, 0);
                nid = j < size ? (lane < 31 ? a : b) : kInvalid;
            } else {
                nid = j < size ? adj[1 + j] : kInvalid;
            }
            uint32_t slot = hash32(nid) & (vc - 1);
            bool fresh = j < size && s.vis[slot] != nid;
            __syncwarp();
            uint32_t fb = __ballot_sync(0xFFFFFFFFu, fresh);
            uint32_t cnt = __popc(fb);
            if (fresh) {
                s.ni[__popc(fb & lanemask_lt())] = nid;
                s.vis[slot] = nid;
            }
            __syncwarp();
            if (cnt == 0) continue;
            warp_dist_list<DM, RK>(v, s.q, s.ni, cnt, s.nd);
            c_dist += cnt;
            const bool have = (uint32_t)lane < cnt;
            beam_insert(s, have ? s.nd[lane] : FLT_MAX, have ? s.ni[lane] : kInvalid, have, EF, tsize, cursor, [&](float d, bool ok, uint32_t id, uint32_t pos) {
                if (!short_rows) return;
                c = next_entry(s, d, ok, id, pos, after, at);
                if (c != kInvalid) load_row(v, c, level, row0, row1);
                known = true;
            });
        }
        if (!short_rows) {
            __syncwarp();
            c = first_unexpanded(s, cursor, tsize, found);
        } else {
            if (!known) {  // nothing to insert
                c = after;
                if (c != kInvalid) load_row(v, c, level, row0, row1);
            }
            found = at;
        }
    }
    c_exp += steps;
    return tsize;
}

// ---------------------------------------------------------------------------
// Team search: the warps of a block on one query, for batches too small to fill
// the device (a lone query, the early batches of a construction), where the
// latency of one expansion after the other is all that counts.
// ---------------------------------------------------------------------------

// One row read by a quad of lanes (RK: a width, kRows16 or kRows4): load() puts its
// first elements (all of them for a width) on their way, dist() finishes the row and
// sums; the distance is valid in all four lanes, and every lane of the warp takes
// part.
template <bool FUSED, int RK>
struct QuadRow {
    static constexpr int CH = RK >= 64 ? RK / 16 : 8;  // 16-element blocks in flight
    float4 u[CH];
    __device__ __forceinline__ void load(const DevView& v, const float* x, bool on) {
        const uint32_t nb = RK >= 64 ? RK / 16 : v.nb;
        const float4* x4 = reinterpret_cast<const float4*>(x) + (threadIdx.x & 3);
#pragma unroll
        for (int k = 0; k < CH; ++k)
            if (on && (RK >= 64 || k < nb)) u[k] = __ldg(x4 + 4 * k);
    }
    __device__ __forceinline__ float dist(const DevView& v, const float* q, const float* x) {
        const uint32_t nb = RK >= 64 ? RK / 16 : v.nb;
        const float4* q4 = reinterpret_cast<const float4*>(q) + (threadIdx.x & 3);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < CH; ++k)
            if (RK >= 64 || k < nb) quad_step<FUSED>(acc, q4[4 * k], u[k]);
        if constexpr (RK < 64) {
            const float4* x4 = reinterpret_cast<const float4*>(x) + (threadIdx.x & 3);
            for (uint32_t i = CH; i < nb; i += CH) {
#pragma unroll
                for (int k = 0; k < CH; ++k)
                    if (i + k < nb) u[k] = __ldg(x4 + 4 * (i + k));
#pragma unroll
                for (int k = 0; k < CH; ++k)
                    if (i + k < nb) quad_step<FUSED>(acc, q4[4 * (i + k)], u[k]);
            }
        }
        return quad_sum16(acc[0], acc[1], acc[2], acc[3]);
    }
};

template <bool FUSED>
struct QuadRow<FUSED, kRows4> {
    static constexpr int CH = 16;  // elements of this lane's accumulator in flight
    float u[CH];
    __device__ __forceinline__ void load(const DevView& v, const float* x, bool on) {
        const uint32_t n4 = v.dim >> 2;
        const float* xc = x + (threadIdx.x & 3);
#pragma unroll
        for (int k = 0; k < CH; ++k)
            if (on && k < n4) u[k] = __ldg(xc + 4 * k);
    }
    __device__ __forceinline__ float dist(const DevView& v, const float* q, const float* x) {
        const uint32_t n4 = v.dim >> 2;
        const int c = threadIdx.x & 3, b = threadIdx.x & 28;
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < CH; ++k)
            if (k < n4) a = sq_step(a, q[4 * k + c] - u[k], FUSED);
        for (uint32_t i = CH; i < n4; i += CH) {
#pragma unroll
            for (int k = 0; k < CH; ++k)
                if (i + k < n4) u[k] = __ldg(x + 4 * (i + k) + c);
#pragma unroll
            for (int k = 0; k < CH; ++k)
                if (i + k < n4) a = sq_step(a, q[4 * (i + k) + c] - u[k], FUSED);
        }
        float s = __shfl_sync(0xFFFFFFFFu, a, b);
#pragma unroll
        for (int k = 1; k < 4; ++k) s = __fadd_rn(s, __shfl_sync(0xFFFFFFFFu, a, b + k));
        return s;
    }
};

__device__ __forceinline__ void touch(const uint32_t* p) {
    asm volatile("{\n .reg .u32 w;\n ld.global.nc.u32 w, [%0];\n}" ::"l"(p));
}

// The level-0 link row of `node`, towards L1: the quad's lanes read one word of each
// of its 32-byte sectors.
__device__ __forceinline__ void quad_touch_links(const DevView& v, uint32_t node) {
    const uint32_t* row = v.adj0 + (size_t)node * v.W0;
    const uint32_t at = 8 * (threadIdx.x & 3);
    if (at < v.W0) touch(row + at);
    if (at == 0) touch(row + v.W0 - 1);
}

// beam_search by a block of kTeamWarps warps (link rows of at most 33 words, EF <= 32
// BB): the same beam.  The first four warps score an expansion's neighbours, eight
// each and one per quad, so the rows cost one round trip; the last one keeps the
// beam, in registers (entry k in lane k mod 32, distances as their bits, which
// order as they do).  One barrier a step: after it every warp knows the scored
// neighbours of the step (nd, ni, two steps' worth), the beam's farthest entry and
// its first unexpanded one as the step before left them (pub), and so the entry
// that is expanded next.  The scoring warps fetch that entry's neighbours at once,
// while the last warp inserts the scored ones.  This needs neighbours that were
// never scored before (one that is in the beam already would be taken for the next
// entry and expanded again, without end): the visited ids are an open-address set
// here, up to three quarters of its vc slots.  A search that goes on from there
// keeps the beam in shared memory, uses the slots as beam_search's lossy cache, and
// its steps wait until the beam is updated.  The link rows of the neighbours that
// are scored, and of the first unexpanded entry, are drawn into L1, where the next
// entry's is then found.
//
// ep and epd are read in warp 0.  ids2: 64 words of shared memory.
constexpr int kTeamWarps = 5;
constexpr uint32_t kTeamMaxEf = 512;

// Searches per SM up to which a batch gets a team each (HRNN_TEAM overrides it, 0:
// never).  At 333 queries of d = 100 teams took 0.58 ms and single warps 0.75 ms; the
// 100k x 128 build took 350 ms with teams up to 4 points per SM, 356 up to 2, 433 up
// to 8, 406 without.
inline size_t team_searches(int nsm) {
    const char* e = std::getenv("HRNN_TEAM");
    return (size_t)nsm * (e ? std::strtoul(e, nullptr, 10) : 4);
}
constexpr uint32_t kNoDist = 0xFFFFFFFFu;  // above every distance's bits

// Slots of a team's visited set: a search at beam efc visits about 12 ids per entry.
inline uint32_t team_vis(uint32_t efc) { return efc <= 128 ? 4096 : 8192; }

// The last warp's beam: BB entries per lane.
template <int BB>
struct RegBeam {
    uint32_t d[BB], i[BB];  // kNoDist / kInvalid beyond the entries
    __device__ __forceinline__ void start(uint32_t d0, uint32_t i0) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int u = 0; u < BB; ++u) d[u] = i[u] = kNoDist;
        if (lane == 0) {
            d[0] = d0;
            i[0] = i0;
        }
    }
    // (x, y) before the first entry farther than x
    __device__ __forceinline__ void insert(uint32_t x, uint32_t y) {
        const int lane = threadIdx.x & 31;
        uint32_t rd = 0, ri = 0;  // lane 0: the last entry of the block before
#pragma unroll
        for (int u = 0; u < BB; ++u) {
            const uint32_t pd = __shfl_sync(0xFFFFFFFFu, d[u], (lane + 31) & 31);
            const uint32_t pi = __shfl_sync(0xFFFFFFFFu, i[u], (lane + 31) & 31);
            const uint32_t bd = lane == 0 ? rd : pd, bi = lane == 0 ? ri : pi;  // the entry before this one
            rd = pd;
            ri = pi;
            const bool after = d[u] > x;
            const bool first = after && (!(bd > x) || (u == 0 && lane == 0));
            d[u] = after ? (first ? x : bd) : d[u];
            i[u] = after ? (first ? y : bi) : i[u];
        }
    }
    __device__ __forceinline__ void cut(uint32_t EF) {
#pragma unroll
        for (int u = 0; u < BB; ++u)
            if (32 * u + (threadIdx.x & 31) >= EF) d[u] = i[u] = kNoDist;
    }
    __device__ __forceinline__ void mark(uint32_t at) {
#pragma unroll
        for (int u = 0; u < BB; ++u)
            if (32 * u + (threadIdx.x & 31) == at) i[u] |= kExpanded;
    }
    // first unexpanded entry: its id (kInvalid: none), distance and place
    __device__ __forceinline__ uint32_t first(uint32_t& at, uint32_t& fd) const {
        uint32_t id = kInvalid;
#pragma unroll
        for (int u = 0; u < BB; ++u) {
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, !(i[u] & kExpanded));
            if (id == kInvalid && bal) {  // uniform
                at = 32 * u + __ffs(bal) - 1;
                id = __shfl_sync(0xFFFFFFFFu, i[u], __ffs(bal) - 1);
                fd = __shfl_sync(0xFFFFFFFFu, d[u], __ffs(bal) - 1);
            }
        }
        return id;
    }
    // distance of entry k
    __device__ __forceinline__ uint32_t dist_at(uint32_t k) const {
        uint32_t x = kNoDist;
#pragma unroll
        for (int u = 0; u < BB; ++u) x = 32 * u + (threadIdx.x & 31) == k ? d[u] : x;
        return __reduce_min_sync(0xFFFFFFFFu, x);
    }
    __device__ __forceinline__ void store(const WarpSmem& s, uint32_t n) const {
#pragma unroll
        for (int u = 0; u < BB; ++u) {
            const uint32_t k = 32 * u + (threadIdx.x & 31);
            if (k < n) {
                s.td[k] = __uint_as_float(d[u]);
                s.ti[k] = i[u];
            }
        }
    }
};

template <bool FUSED, int RK, int BB>
__device__ uint32_t beam_search_team(const DevView& v, WarpSmem& s, uint32_t* ids2, uint32_t ep, float epd, uint32_t EF,
                                     int level, uint32_t vc, unsigned long long& c_dist, unsigned long long& c_exp) {
    constexpr uint32_t NT = 32 * kTeamWarps;
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31, w = tid >> 5, c4 = lane & 3, r = lane >> 2;
    const bool keeper = w == kTeamWarps - 1;
    // two steps' worth of: unexpanded entry, its distance, the bits that a neighbour
    // has to be below
    uint32_t* pub = s.apos;
    uint32_t* fresh_n = s.apos + 8;  // ids each warp added to the visited set
    for (uint32_t i = tid; i < vc; i += NT) s.vis[i] = kInvalid;
    if (tid == 0) {
        s.td[0] = epd;
        s.ti[0] = ep;
        pub[0] = kInvalid;  // (read after step 0)
        pub[2] = EF > 1 ? kNoDist : __float_as_uint(epd);
    }
    __syncthreads();
    uint32_t c = s.ti[0], tsize = 1, cursor = 0, at = 0;
    if (tid == 0) s.vis[hash32(c) & (vc - 1)] = c;
    __syncthreads();
    // The keeper's and the scorers' loops meet at the same barriers, step by step; two
    // loops, so that neither's registers weigh on the other.
    uint32_t visited = 1;
    // After a step's scores: the next entry -- the closest neighbour that enters the
    // beam (lane ln of those in `have`), or the first unexpanded entry where none is
    // closer -- and whether the visited set still has room (`exact`).
    struct Next {
        uint32_t c, have;
        int ln;
        bool fromnew, exact;
    };
    auto choose = [&](uint32_t buf, uint32_t d, uint32_t id) {
        const uint4 p = reinterpret_cast<const uint4*>(pub)[buf], n = reinterpret_cast<const uint4*>(fresh_n)[buf];
        visited += n.x + n.y + n.z + n.w;
        Next x;
        const bool ok = d < p.z;
        const uint32_t best = __reduce_min_sync(0xFFFFFFFFu, ok ? d : kNoDist);
        x.have = __ballot_sync(0xFFFFFFFFu, ok);
        x.fromnew = x.have && !(p.x != kInvalid && p.y <= best);
        x.ln = (__ffs(__ballot_sync(0xFFFFFFFFu, ok && d == best)) - 1) & 31;
        const uint32_t cand = __shfl_sync(0xFFFFFFFFu, id, x.ln);
        x.c = x.fromnew ? cand : p.x;
        x.exact = visited + 32 <= vc / 4 * 3;
        return x;
    };
    auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * kTeamWarps) : "memory"); };
    const uint32_t* nd0 = reinterpret_cast<const uint32_t*>(s.nd);  // (s.ni follows s.nd)
    bool exact = true;
    if (keeper) {
        RegBeam<BB> beam;
        c_exp++;
        beam.start(__float_as_uint(s.td[0]), c | kExpanded);
        for (uint32_t step = 0; step <= v.n; ++step) {  // (every step expands another node)
            const uint32_t buf = step & 1;
            meet();
            const uint32_t d = nd0[32 * buf + lane], id = ids2[32 * buf + lane];
            if (exact) {
                const Next x = choose(buf, d, id);
                c = x.c;
                exact = x.exact;
                if (c != kInvalid) c_exp++;
                if (!x.fromnew && c != kInvalid) beam.mark(at);
                const uint32_t y = x.fromnew && lane == x.ln ? id | kExpanded : id;
#pragma unroll 1
                for (uint32_t m = x.have; m; m &= m - 1) {
                    const int j = __ffs(m) - 1;
                    beam.insert(__shfl_sync(0xFFFFFFFFu, d, j), __shfl_sync(0xFFFFFFFFu, y, j));
                }
                if (x.have) {
                    tsize = min(tsize + __popc(x.have), EF);
                    beam.cut(EF);
                }
                if (c != kInvalid && exact) {
                    uint32_t fd = 0;
                    const uint32_t nx = beam.first(at, fd);
                    const uint32_t last = tsize >= EF ? beam.dist_at(EF - 1) : kNoDist;
                    if (lane == 0) reinterpret_cast<uint4*>(pub)[buf ^ 1] = make_uint4(nx, fd, last, 0u);
                    if (nx != kInvalid && level == 0) quad_touch_links(v, nx);
                } else {  // the search ends or goes on in shared memory
                    beam.store(s, tsize);
                    __syncwarp();
                }
            } else {
                beam_insert(s, __uint_as_float(d), id, d != kNoDist, EF, tsize, cursor,
                            [](float, bool, uint32_t, uint32_t) {});
                c = first_unexpanded(s, cursor, tsize, at);
                __syncwarp();
                if (c != kInvalid) {
                    cursor = at + 1;
                    c_exp++;
                    if (lane == 0) s.ti[at] = c | kExpanded;
                }
                if (lane == 0) pub[4 * buf] = c;
                meet();
            }
            if (c == kInvalid) break;
        }
        if (lane == 0) s.apos[16] = tsize;
    } else {
        const uint32_t jq = 8 * w + r;
        for (uint32_t step = 0; step <= v.n; ++step) {
            const uint32_t buf = step & 1;
            // this quad's neighbour of c
            uint32_t w0, w1;
            load_row(v, c, level, w0, w1);
            const uint32_t size = __shfl_sync(0xFFFFFFFFu, w0, 0) & 0xFFFFu;
            const uint32_t a = __shfl_sync(0xFFFFFFFFu, w0, (jq + 1) & 31), z = __shfl_sync(0xFFFFFFFFu, w1, 0);
            const uint32_t id = jq < 31 ? a : z;
            bool fresh = false;
            if (c4 == 0 && jq < size) {
                uint32_t slot = hash32(id) & (vc - 1);
                uint32_t old = s.vis[slot];
                if (exact) {
                    // most neighbours have been met: a read tells, and only a free
                    // slot is worth an atomic (a quarter of them stays free)
                    while (old != id) {
                        if (old == kInvalid) {
                            old = atomicCAS(&s.vis[slot], kInvalid, id);
                            if (old == kInvalid) {
                                fresh = true;
                                break;
                            }
                        } else {
                            slot = (slot + 1) & (vc - 1);
                            old = s.vis[slot];
                        }
                    }
                } else {
                    fresh = old != id;
                    s.vis[slot] = id;
                }
            }
            const uint32_t fb = __ballot_sync(0xFFFFFFFFu, fresh);
            fresh = fb >> (lane & ~3) & 1u;
            uint32_t bits = kNoDist;
            if (fb) {
                const float* x = v.vec + (size_t)(fresh ? id : c) * v.dim;
                QuadRow<FUSED, RK> row;
                row.load(v, x, fresh);
                if (fresh && level == 0) quad_touch_links(v, id);  // (above, the row's place is a read away)
                const float d = row.dist(v, s.q, x);
                if (fresh) bits = __float_as_uint(d);
            }
            if (c4 == 0) {
                s.nd[32 * buf + jq] = __uint_as_float(bits);
                ids2[32 * buf + jq] = id;
            }
            if (lane == 0) {
                fresh_n[4 * buf + w] = __popc(fb);
                c_dist += __popc(fb);
            }
            meet();
            if (exact) {
                const Next x = choose(buf, nd0[32 * buf + lane], ids2[32 * buf + lane]);
                c = x.c;
                exact = x.exact;
            } else {
                meet();
                c = pub[4 * buf];
            }
            if (c == kInvalid) break;
        }
    }
    __syncthreads();
    tsize = s.apos[16];
    __syncthreads();
    return tsize;
}

}  // namespace hrnn
