// One warp on the host: 32 fibers that meet at every warp-wide operation, so that the
// warp-level device functions can be compiled by g++ and checked without a GPU.
#pragma once

#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include <cuda_runtime.h>

namespace hostwarp {

struct Lane {
    ucontext_t ctx;
    std::vector<char> stack = std::vector<char>(1 << 17);
    bool done = false;
    unsigned ops = 0;
};
inline Lane lanes[32];
inline ucontext_t back;
inline uint64_t slot[2][32];  // the lanes' operands of this operation and of the next
inline std::function<void()> body;
struct Idx {
    unsigned x = 0;
} inline here;

inline void enter() {
    body();
    lanes[here.x].done = true;
    swapcontext(&lanes[here.x].ctx, &back);
}

// Every lane runs f; false when it has not ended after `limit` warp-wide operations.
inline bool run(std::function<void()> f, uint64_t limit) {
    body = std::move(f);
    for (Lane& l : lanes) {
        l.done = false;
        l.ops = 0;
        getcontext(&l.ctx);
        l.ctx.uc_stack.ss_sp = l.stack.data();
        l.ctx.uc_stack.ss_size = l.stack.size();
        l.ctx.uc_link = nullptr;
        makecontext(&l.ctx, (void (*)())enter, 0);
    }
    for (uint64_t op = 0; op < limit; ++op) {
        unsigned ended = 0;
        for (unsigned i = 0; i < 32; ++i) {
            here.x = i;
            if (!lanes[i].done) swapcontext(&back, &lanes[i].ctx);
            ended += lanes[i].done;
        }
        if (ended == 32) return true;
        if (ended) {
            std::fprintf(stderr, "lanes ended in different operations\n");
            std::abort();
        }
    }
    return false;
}

// All lanes' operands, once every lane has come here.
inline const uint64_t* meet(uint64_t v) {
    const unsigned i = here.x, p = lanes[i].ops++ & 1;
    slot[p][i] = v;
    swapcontext(&lanes[i].ctx, &back);
    return slot[p];
}

template <class T>
uint64_t pack(T v) {
    uint64_t r = 0;
    std::memcpy(&r, &v, sizeof v);
    return r;
}
template <class T>
T unpack(uint64_t r) {
    T v;
    std::memcpy(&v, &r, sizeof v);
    return v;
}

}  // namespace hostwarp

#define threadIdx (hostwarp::here)
#define asm(...) m = (1u << hostwarp::here.x) - 1u  // %lanemask_lt

inline void __syncwarp() { hostwarp::meet(0); }
inline void __syncthreads() { std::abort(); }  // (one warp)
inline uint32_t __ballot_sync(uint32_t, bool b) {
    const uint64_t* o = hostwarp::meet(b);
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= (uint32_t)o[i] << i;
    return r;
}
template <class T>
T __shfl_sync(uint32_t, T v, int src, int width = 32) {
    const unsigned base = threadIdx.x & ~(width - 1u);
    return hostwarp::unpack<T>(hostwarp::meet(hostwarp::pack(v))[base + (src & (width - 1))]);
}
template <class T>
T __shfl_xor_sync(uint32_t, T v, int x) {
    return hostwarp::unpack<T>(hostwarp::meet(hostwarp::pack(v))[threadIdx.x ^ x]);
}
template <class T>
T __shfl_down_sync(uint32_t, T v, int x) {
    const unsigned i = threadIdx.x;
    return hostwarp::unpack<T>(hostwarp::meet(hostwarp::pack(v))[i + x < 32 ? i + x : i]);
}
inline uint32_t __reduce_min_sync(uint32_t, uint32_t v) {
    const uint64_t* o = hostwarp::meet(v);
    uint32_t r = 0xFFFFFFFFu;
    for (int i = 0; i < 32; ++i) r = o[i] < r ? (uint32_t)o[i] : r;
    return r;
}
inline uint32_t __match_any_sync(uint32_t, uint32_t v) {
    const uint64_t* o = hostwarp::meet(v);
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= (uint32_t)(o[i] == v) << i;
    return r;
}
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
inline uint32_t __float_as_uint(float x) { return (uint32_t)hostwarp::pack(x); }
inline float __uint_as_float(uint32_t x) { return hostwarp::unpack<float>(x); }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float __double2float_ru(double a) {
    const float f = (float)a;
    return (double)f < a ? std::nextafterf(f, INFINITY) : f;
}
inline int __float2int_rn(float a) { return (int)std::nearbyintf(a); }
template <class T>
T __ldg(const T* p) { return *p; }
inline int __dp4a(int a, int b, int c) {
    for (int i = 0; i < 4; ++i) c += (int)(int8_t)(a >> 8 * i) * (int)(int8_t)(b >> 8 * i);
    return c;
}
inline uint32_t atomicCAS(uint32_t* p, uint32_t a, uint32_t b) {
    const uint32_t o = *p;
    if (o == a) *p = b;
    return o;
}
template <class T>
T min(T a, T b) { return b < a ? b : a; }
template <class T>
T max(T a, T b) { return a < b ? b : a; }
inline int min(int a, int b) { return b < a ? b : a; }
