// gde_device.cuh -- small device helpers shared by the kernel translation units.
#pragma once
#include <cstdint>

#include "gde_common.cuh"

namespace gde {

constexpr unsigned long long kSpinLimit = 1ull << 26;  // ~ seconds of polling

// ---------------------------------------------------------------------------
// Bounded grid barrier (a counter of arrivals).  Co-residency of all
// blocks is guaranteed by the cooperative launch; the spin limit only guards
// against a bug turning into a hang: on expiry the block records GDE_EHANG
// and every block leaves its loop at the next barrier.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int ld_volatile_i(const int* p) { return *(volatile const int*)p; }
// A load that later loads of this thread cannot pass (device-scope acquire).
__device__ __forceinline__ int ld_acquire_gpu_i(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long ld_acquire_gpu_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long add_release_gpu_u64(unsigned long long* p, unsigned long long x) {
    unsigned long long v;
    asm volatile("atom.add.release.gpu.u64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(x) : "memory");
    return v;
}

// `limit` polls (0: kSpinLimit) before a waiting block gives up; `members`
// blocks meet at `bar` (0: the whole grid).  Arrivals only count up, so a
// block knows from its own ticket the count that completes its phase and
// polls for it: one release, one round trip for the ticket and one for the
// last arrival, with no second word to reset and publish (2.8 us of a round's
// ~23 on a small graph before, twice a round).
__device__ __forceinline__ bool grid_barrier(GridBarrier* bar, int* err, unsigned long long limit = 0,
                                             unsigned members = 0) {
    if (limit == 0) limit = kSpinLimit;
    if (members == 0) members = gridDim.x;
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned long long ticket = add_release_gpu_u64(&bar->count, 1ull);
        const unsigned long long target = (ticket / members + 1) * members;
        unsigned long long spins = 0;
        for (;;) {
            const int e = ld_volatile_i(err);  // in flight with the count
            const bool all = ld_acquire_gpu_u64(&bar->count) >= target;
            if (e != 0) ok = 0;
            if (all || e != 0) break;
            if (++spins > limit) {
                atomicCAS(err, 0, GDE_EHANG);
                ok = 0;
                break;
            }
            __nanosleep(32);
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Device-wide nanosecond clock (PTX %globaltimer).
__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// FP64 comparisons |r| >= thr and r >= thr of a threshold thr >= 0, on the
// bit patterns (the order of non-negative doubles is that of their bits; a
// NaN compares false, as in FP64).  GB300 runs one FP64 instruction per SM
// and warp in 16 cycles, an integer one in one: the FP64 tiles' tests, like
// their divisions (DevGraph::rdeg), stay off that pipe where they can.
constexpr long long kInfBits = 0x7ff0000000000000ll;
__device__ __forceinline__ bool ge_bits(long long r, long long thr) { return r >= thr && r <= kInfBits; }
__device__ __forceinline__ bool ge_abs64(double r, double thr) {
    return ge_bits(__double_as_longlong(r) & 0x7fffffffffffffffll, __double_as_longlong(thr));
}

// A work item of a one-column tile holds its push value instead of the
// frontier index of a push row: the edges are one load away from the item.
// Row starts take 40 bits and lengths 24 (the host caps the row classes).
// FP32 items of a merged leaf hold its own push value and `times` it is pushed
// (with its twins'); 0: once.
template <typename T>
__device__ __forceinline__ PushItem pack_item(long long rp, int len, T push, int times = 0) {
    PushItem it;
    it.rp = rp | ((long long)len << 40);
    if constexpr (sizeof(T) == 8) {
        it.len = __double2hiint(push);
        it.node = __double2loint(push);
    } else {
        it.len = times;
        it.node = __float_as_int(push);
    }
    return it;
}
// The sum that an FP32 item of one edge pushes, whole: 24 bits times up to 23 fit
// FP64's 53.  In integers: FP64 instructions issue at 1/16 rate.
__device__ __forceinline__ double item_sum(const PushItem& it) {
    const unsigned b = (unsigned)it.node, e = b >> 23 & 0xffu, times = it.len > 1 ? it.len : 1;
    if (e == 0u || e == 0xffu) return (double)__int_as_float(it.node) * times;
    const unsigned long long p = (unsigned long long)((b & 0x7fffffu) | 0x800000u) * times;
    const int z = __clzll((long long)p);  // the product's first bit is 63 - z; 24 bits alone would be at 23
    return __longlong_as_double((long long)((unsigned long long)(b >> 31) << 63 |
                                            (unsigned long long)(e + 1023 - 127 + 40 - z) << 52 | p << (z + 1) >> 12));
}
template <typename T>
__device__ __forceinline__ T unpack_item(const PushItem& it, long long& rp, int& len) {
    rp = it.rp & ((1ll << 40) - 1);
    len = (int)((unsigned long long)it.rp >> 40);
    if constexpr (sizeof(T) == 8) return __hiloint2double(it.len, it.node);
    else return __int_as_float(it.node);
}

// Append v to a candidate list once per stamp (mark dedup), one atomic per
// warp for all appending lanes.  `mask` must name every lane executing the
// call.
__device__ __forceinline__ void append_once(bool want, int v, int32_t* mark, int stamp, int32_t* list, int* cnt,
                                            unsigned mask) {
    bool app = false;
    if (want) {
        if (mark[v] != stamp) app = (atomicExch(&mark[v], stamp) != stamp);
    }
    unsigned b = __ballot_sync(mask, app);
    if (b) {
        int lane = threadIdx.x & 31;
        int leader = __ffs(b) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(cnt, __popc(b));
        base = __shfl_sync(mask, base, leader);
        if (app) list[base + __popc(b & ((1u << lane) - 1u))] = v;
    }
}

}  // namespace gde
