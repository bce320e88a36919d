// Adding rows into a large buffer whose rows are touched in random order: the work sorted into
// BINS (ranges of the buffer that fit the L2 several times), taken bin after bin by the whole
// grid, with every bin cleared shortly before it is added to.  A line of the buffer is then
// written to DRAM once and never read, where clearing first and adding in random order costs two
// writes and a read.
#pragma once

#include "common.cuh"

namespace svoxb {

constexpr int kMaxBins = 128;
// Floats a block clears at a time.  Measured (scatter of 2^24 query rows, of an 800x800 SH16 view,
// of se_grad for 100000 rays, of 2^20 rays; ms): 8192: 2.86, 1.44, 1.13, 1.86; 16384: 2.60, 1.35,
// 1.13, 1.86; 65536: 2.40, 1.30, 1.10, 1.88.
constexpr int kZeroFloats = 65536;

// L2 residency hints.
__device__ __forceinline__ uint64_t l2_policy_keep() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_stream() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void st_hint16(void* a, int4 v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.v4.s32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(a), "r"(v.x),
                 "r"(v.y), "r"(v.z), "r"(v.w), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void red_add_v4_hint(float* addr, float a, float b, float c, float d,
                                                uint64_t pol) {
    asm volatile("red.global.add.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(addr),
                 "f"(a), "f"(b), "f"(c), "f"(d), "l"(pol)
                 : "memory");
}

// Counters of one launch, in global memory, all zero before it; the last block puts them back.
struct UnitCounters {
    int32_t* next;       // units taken
    int32_t* done;       // blocks done
    int32_t* cleared;    // [n_bins] units of clearing done per bin
};

struct UnitShared {
    int start[kMaxBins + 1];    // first unit of bin b
    int first[kMaxBins + 1];    // its first item
    int zero[kMaxBins + 1];     // its units of clearing
    int unit, bin, place;
};

// Works through the bins [lo, hi): `count(b)` items of bin b, the items of all bins numbered
// through from `before` on; a unit is up to `per_unit` of a bin's items, handed to
// `work(first, end)` by all threads of the block.  With `clear_floats` > 0 (the length of the
// outputs) bin b + 1, `bin_floats` floats, is cleared by `clear(from, until)` in units that come
// before the items of bin b, the first bin before all; with `spread` they are spread over the first
// two thirds of the bin's units instead, so that clearing and adding run side by side: worth while
// where units are large, in the middle of the lengths that were tried, see the call in
// render_replay.cuh.
//
// Units are taken by blocks in order from one counter, so that the grid works within a window
// much smaller than a bin (with a fixed assignment the blocks drift apart and several bins compete
// for the L2: 2.9 ms for the scatter of 2^20 rays against 1.7 in this order, then; with a unit per
// warp the counter itself is the bound, some 6 ns per unit).  A unit may have to wait for the
// clearing of its bin: those units were all taken before it, and a block works on its units in
// order, so the oldest unit that is not done never waits.
template <int BLOCK, class Count, class Clear, class Work>
__device__ __forceinline__ void ordered_units(UnitShared& s, const UnitCounters& counters, int lo,
                                              int hi, int before, int per_unit, int64_t bin_floats,
                                              int64_t clear_floats, bool spread, Count count,
                                              Clear clear, Work work) {
    for (int b = threadIdx.x; b <= kMaxBins; b += BLOCK) {
        const int64_t left = clear_floats - b * bin_floats;
        s.zero[b] = clear_floats > 0 && b < hi && left > 0
                        ? (int)(((left < bin_floats ? left : bin_floats) + kZeroFloats - 1) / kZeroFloats)
                        : 0;
        s.first[b] = b >= lo && b < hi ? count(b) : 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int item = before, unit = s.zero[lo];
        for (int b = lo; b < hi; ++b) {
            const int n = s.first[b];
            s.start[b] = unit;
            s.first[b] = item;
            unit += s.zero[b + 1] + (n + per_unit - 1) / per_unit;
            item += n;
        }
        s.start[hi] = unit;
        s.first[hi] = item;
    }
    __syncthreads();
    const int all = s.start[hi], head = s.zero[lo];
    int taken = 0, at_bin = lo, ready = -1;     // thread 0; `ready`: bin known to be cleared
    if (threadIdx.x == 0) taken = atomicAdd(counters.next, 1);
    for (;;) {
        if (threadIdx.x == 0) {
            int bin = lo, u = taken, z = head;              // clearing of the first bin
            if (taken >= head && taken < all) {
                while (taken >= s.start[at_bin + 1]) ++at_bin;     // a block's units ascend
                bin = at_bin;
                u = taken - s.start[bin];
                z = s.zero[bin + 1];
                int before = u < z ? u : z, upto = u < z ? u + 1 : z;    // units of clearing
                if (spread && z > 0) {
                    const int n = s.start[bin + 1] - s.start[bin];
                    const int64_t num = 3 * z < 2 * n ? 3 * z : 2 * n;
                    before = (int)min((int64_t)z, u * num / (2 * n));
                    upto = (int)min((int64_t)z, (u + 1) * num / (2 * n));
                }
                if (before < upto) {
                    ++bin;
                    u = before;
                } else {
                    z = before;
                    if (clear_floats > 0 && bin != ready) {
                        int tries = 0;
                        while (*(volatile int32_t*)(counters.cleared + bin) < s.zero[bin] &&
                               ++tries < (1 << 22))
                            __nanosleep(64);
                        if (tries == (1 << 22)) report(SVOXB_ERR_CUDA);
                        __threadfence();
                        ready = bin;
                    }
                }
            }
            s.unit = taken;
            s.bin = bin;
            s.place = u - z;
        }
        __syncthreads();
        const int bin = s.bin, place = s.place;
        if (s.unit >= all) break;
        if (threadIdx.x == 0) taken = atomicAdd(counters.next, 1);   // arrives during this unit
        if (place < 0) {
            const int64_t from = bin * bin_floats + (int64_t)(place + s.zero[bin]) * kZeroFloats;
            int64_t until = from + kZeroFloats;
            if (until > (bin + 1) * bin_floats) until = (bin + 1) * bin_floats;
            if (until > clear_floats) until = clear_floats;
            clear(from, until);
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(counters.cleared + bin, 1);
            }
            continue;
        }
        work(s.first[bin] + place * per_unit, s.first[bin + 1]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(counters.done, 1) == (int)gridDim.x - 1) {
            *counters.next = 0;
            *counters.done = 0;
            for (int b = lo; b < hi; ++b) counters.cleared[b] = 0;
        }
    }
}

}  // namespace svoxb
