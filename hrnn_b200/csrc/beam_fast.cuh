// Two-parent best-first search of level 0 for the reduced-precision search forms
// (INT8 / BF16 rows).  Their proxies only choose candidates -- every returned
// point is decided exactly afterwards -- so this search is free to differ from
// searchBaseLayerST's sequential order (hrnn.h:484-616), which the exact form's
// beam.cuh keeps:
//
//   * each step expands the two best unexpanded beam entries together: both link
//     rows are loaded at once and all their fresh neighbours (up to 64) are
//     scored in one memory round trip (INT8 rows read by eight lanes each), so a step costs
//     one dependent row-gather latency for two expansions;
//   * a scored neighbour enters the beam when it is closer than a full beam's last
//     entry (no per-neighbour sequential acceptance count), duplicates within a
//     step are merged with __match_any_sync, duplicates of beam entries by the
//     equal-distance check;
//   * the beam can be saved after a search with a small beam and resumed later
//     with a larger one (the learned budget's fallback continues the frontier
//     search instead of starting over).
// The search ends when no unexpanded entry is left in the beam, like the
// reference's stop rule (cand_dist > lowerBound with a full result heap).
#pragma once

#include "beam.cuh"

namespace hrnn {

// Per-warp shared memory of the two-parent search:
// q | q8 (dim bytes, padded to 16) | qm | td[efc+32] | ti[efc+32] | vis[vc] | nd[64] | ni[64] | apos[32]
__host__ __device__ inline size_t fast_smem_bytes(uint32_t dim, uint32_t efc, uint32_t vc) {
    return (size_t)dim * 4 + (((size_t)dim + 15) & ~(size_t)15) + 16 + (size_t)(efc + 32) * 8 + (size_t)vc * 4 +
           64 * 8 + 32 * 4;
}

__device__ inline WarpSmem carve_fast(char* base, uint32_t dim, uint32_t efc, uint32_t vc) {
    WarpSmem s;
    s.q = (float*)base;
    base += (size_t)dim * 4;
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
    base += 64 * 4;
    s.ni = (uint32_t*)base;
    base += 64 * 4;
    s.apos = (uint32_t*)base;
    return s;
}

// 32 rows' reads on their way, eight lanes per row (coop_i8_load): four whole rows per
// load instruction; rows of 256 bytes in two halves.
template <int NB>
struct CoopRows {
    static constexpr int H = NB > 8 ? 2 : 1;
    int4 x[H][8];
    float4 m;
    __device__ __forceinline__ void load(const DevView& v, const uint32_t* ids, uint32_t b0, uint32_t cnt) {
        const int g = (threadIdx.x >> 3) & 3;
        const uint32_t r = coop_row();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t t = b0 + 4 * i + g;
            const uint32_t id = ids[t < cnt ? t : 0];
            if constexpr (H == 1) {
                x[0][i] = coop_i8_load<NB>(v.vec_i8, id);
            } else {
                const int4* row = reinterpret_cast<const int4*>(v.vec_i8 + (size_t)id * (NB * 16)) + (threadIdx.x & 7);
                x[0][i] = __ldg(row);
                x[1][i] = __ldg(row + 8);
            }
        }
        m = __ldg(v.i8_meta + ids[b0 + r < cnt ? b0 + r : 0]);
    }
    __device__ __forceinline__ void score(const int4 (&qw)[H], float4 qm, uint32_t b0, uint32_t cnt, float* dout) const {
        int p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            p[i] = dp4a4(x[0][i], qw[0]);
            if constexpr (H == 2) p[i] += dp4a4(x[1][i], qw[1]);
        }
        const int d = coop_sum8(p);
        const uint32_t r = coop_row();
        if (b0 + r < cnt) dout[b0 + r] = qm.x + m.x * m.x * m.z - 2.f * qm.y * m.x * (float)d;
    }
};

// ids[0..cnt) (cnt <= 64) scored with cooperative row reads, 32 at a time.  R2: both
// blocks' loads issued before either is scored (one memory round trip for 64 rows,
// twice the registers); otherwise block by block.
template <int NB, bool R2>
__device__ __forceinline__ void warp_i8_coop(const DevView& v, const int* q8, float4 qm, const uint32_t* ids,
                                             uint32_t cnt, float* dout) {
    int4 qw[CoopRows<NB>::H];
    qw[0] = coop_q_words<(NB > 8 ? 8 : NB)>(q8);
    if constexpr (NB > 8) qw[1] = coop_q_words<8>(q8 + 32);
    if constexpr (R2) {
        CoopRows<NB> a, b;
        a.load(v, ids, 0, cnt);
        if (cnt > 32) b.load(v, ids, 32, cnt);
        a.score(qw, qm, 0, cnt, dout);
        if (cnt > 32) b.score(qw, qm, 32, cnt, dout);
    } else {
        for (uint32_t b0 = 0; b0 < cnt; b0 += 32) {
            CoopRows<NB> a;
            a.load(v, ids, b0, cnt);
            a.score(qw, qm, b0, cnt, dout);
        }
    }
}

// Scores ids[0..cnt) (cnt <= 64) with the form's rows: DM 3 INT8, DM 2 BF16.
// R2: all 64 rows in one memory round trip (at more registers and so fewer resident
// warps; two at 256 BF16 elements) or 32 INT8 / 16 BF16 rows at a time; the launch-shape
// autotuner picks for INT8, and small batches, where latency counts, take R2.
// RK: the width (0: any).
template <int DM, bool R2, int RK>
__device__ __forceinline__ void warp_dist_list64(const DevView& v, const float* q, const uint32_t* ids,
                                                 uint32_t cnt, float* dout) {
    // INT8 rows of 96, 128 and 256 bytes read cooperatively; other widths one row per
    // lane, 32 at a time
    if constexpr (DM == 3 && RK >= 64) {
        warp_i8_coop<RK / 16, R2>(v, i8_q_words(q, RK), *i8_q_meta(q, RK), ids, cnt, dout);
        __syncwarp();
    } else if constexpr (DM == 2 && RK >= 64 && R2) {
        warp_bf16_pairs<RK / 16, RK <= 128 ? 4 : 2>(v, q, ids, cnt, dout);
        __syncwarp();
    } else {
        warp_dist_list<DM, RK>(v, q, ids, min(cnt, 32u), dout);
        if (cnt > 32) warp_dist_list<DM, RK>(v, q, ids + 32, cnt - 32, dout + 32);
    }
}

// Two-parent search of level 0 continuing from the beam s.td/s.ti[0..tsize)
// (sorted; ids carry kExpanded).  The visited cache must hold (at least) the
// beam's ids.  The beam keeps the EF nearest scored points; only its first EX
// (<= EF) are expanded, the rest is a reserve a later search with a larger beam
// can resume from (the first EX entries evolve exactly as in a search with
// EF = EX).  Returns the beam size (<= EF).
template <int DM, bool R2, int RK>
__device__ uint32_t beam_search_fast(const DevView& v, WarpSmem& s, uint32_t tsize, uint32_t EF, uint32_t EX,
                                     uint32_t vc, unsigned long long& c_dist, unsigned long long& c_exp) {
    const int lane = threadIdx.x & 31;
    uint32_t cursor = 0;
    for (;;) {
        // the (up to) two best unexpanded entries at or after cursor, among the first EX
        uint32_t par0 = kInvalid, par1 = kInvalid;
        const uint32_t lim = min(tsize, EX);
        for (uint32_t b = cursor; b < lim; b += 32) {
            const uint32_t idx = b + lane;
            const bool u = idx < lim && !(s.ti[idx] & kExpanded);
            uint32_t bal = __ballot_sync(0xFFFFFFFFu, u);
            if (!bal) continue;
            if (par0 == kInvalid) {
                par0 = b + __ffs(bal) - 1;
                bal &= bal - 1;
            }
            if (bal) {
                par1 = b + __ffs(bal) - 1;
                break;
            }
        }
        if (par0 == kInvalid) break;
        const uint32_t c0 = s.ti[par0] & kIdMask;
        const uint32_t c1 = par1 != kInvalid ? (s.ti[par1] & kIdMask) : kInvalid;
        cursor = (par1 != kInvalid ? par1 : par0) + 1;
        __syncwarp();
        if (lane == 0) {
            s.ti[par0] |= kExpanded;
            if (par1 != kInvalid) s.ti[par1] |= kExpanded;
        }
        c_exp += par1 != kInvalid ? 2 : 1;
        // both link rows in one go (rows of at most 33 words, maxM0 <= 32)
        uint32_t ra0 = 0, ra1 = 0, rb0 = 0, rb1 = 0;
        load_row(v, c0, 0, ra0, ra1);
        if (c1 != kInvalid) load_row(v, c1, 0, rb0, rb1);
        uint32_t cnt = 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t w0 = r ? rb0 : ra0, w1 = r ? rb1 : ra1;
            const uint32_t size = r && c1 == kInvalid ? 0u : (__shfl_sync(0xFFFFFFFFu, w0, 0) & 0xFFFFu);
            const uint32_t a = __shfl_sync(0xFFFFFFFFu, w0, (lane + 1) & 31);
            const uint32_t bw = __shfl_sync(0xFFFFFFFFu, w1, 0);
            const uint32_t nid = (uint32_t)lane < size ? (lane < 31 ? a : bw) : kInvalid;
            const uint32_t slot = hash32(nid) & (vc - 1);
            const bool fresh = (uint32_t)lane < size && s.vis[slot] != nid;
            __syncwarp();
            const uint32_t fb = __ballot_sync(0xFFFFFFFFu, fresh);
            if (fresh) {
                s.ni[cnt + __popc(fb & lanemask_lt())] = nid;
                s.vis[slot] = nid;
            }
            cnt += __popc(fb);
            __syncwarp();
        }
        if (cnt == 0) continue;
        warp_dist_list64<DM, R2, RK>(v, s.q, s.ni, cnt, s.nd);
        c_dist += cnt;
        for (uint32_t b = 0; b < cnt; b += 32) {
            const bool have = b + lane < cnt;
            beam_insert<true>(s, have ? s.nd[b + lane] : FLT_MAX, have ? s.ni[b + lane] : kInvalid, have, EF, tsize,
                              cursor, [](float, bool, uint32_t, uint32_t) {});
        }
    }
    return tsize;
}

}  // namespace hrnn
