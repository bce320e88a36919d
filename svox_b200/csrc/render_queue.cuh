// Queue-based warp-cooperative volume rendering for octrees (N = 2) whose records hold three
// colour channels: K = 3 * basis_dim + 1 floats, or RGBA with K = 4 (BD = 0 here).  Forward, and
// forward with an item log (the marching backward: render_back.cuh).
//
//   G step  one lane = one ray.  Every iteration takes one SAMPLE per lane: the leaf is found
//           by one table look-up, or one brick look-up below it (render_index.cuh), whose entry
//           already holds the leaf's density, so the march itself reads L2-resident index
//           entries only.  A contributing sample is pushed as an ITEM (leaf slot, optical depth,
//           owner) into the warp's queue in shared memory.
//   S step  one lane = one item.  When 32 items are queued their records are requested with
//           cp.async (coalesced 16-byte words, global -> shared staging rows) and the warp
//           goes on marching; the batch is evaluated when the next one is full, by which time
//           the data has arrived.  Lane i evaluates item i (attenuation, dot products with the
//           owner ray's colour basis, sigmoids); then every owner folds the results of its own items into
//           its ray's transmittance and sums in march order, which keeps the reference's order of accumulation
//           (svox/csrc/rt_kernel.cu:282-295) whatever the batches are.
//
// Bound: issue slots where neighbouring rays share records (images: 61 % of the slots used), DRAM
// too where every sample's record misses (rays in random order: 16 GB for 2^20 rays of the 512^3
// shell scene).  So the march is kept short: an 800x800 view of the shell scene with SH16 records takes
// 0.504 G warp instructions: 2.28 M iterations of 94, 0.49 M batches of items at 390 (325 with 9 logged
// functions), the rest pushes and refills.  The leaf's corner
// comes from truncating additions, its exit distance from five operations per axis, two axes to
// an instruction; lanes between samples compute along instead of branching; the index entry of a
// sample is requested one iteration ahead so that the queue's work covers its latency; and a block holds
// four warps so that shared memory and the L1 can be balanced (kMarchBlocks).
//
// What the march's instructions were, and what became of them (0.583 G before; 15 % of them were
// branches and their reconvergence, 9 % constants and addresses worked out again):
//  - the early stop summed as optical depth, where it was an exponential and a branch per sample;
//  - one word for a lane's state and the samples it has left; seldom cases behind one vote;
//  - items in one or two stores; the product of length and density formed by the march's lanes;
//  - index entries addressed in bytes, by masks that the host works out;
//  - nothing of a ray's set-up or of the log's layout kept in registers through the march (the
//    compiler moved it out of the loop, then spilled: the logged SH9 march 16 % slower), and the
//    lane, the queue's place and the policy not worked out again.
// us before and after, whole call: 800x800 view, SH16 1133 and 1044, SH4 859 and 762, SH9 with
// thresholds 757 and 660; 65536 RGBA rays with gradient 233 and 218; 2^20 SH9 rays with gradient
// 5640 and 5566 (bound by memory); four 1080p views of the 1024^3 scene 20.2 and 18.6 ms.  (Dot
// products with two coefficients per instruction: level for SH9 to SH25.)
//
// Lanes whose ray has ended wait until `refill` of them do; then the queue is drained, their
// results are written and they take new rays from a block-wide ticket counter together (the
// set-up of a ray is some 300 instructions that the whole warp issues).  All control flow
// around warp-level primitives is driven by votes.
#pragma once

#include "render.cuh"
#include "render_index.cuh"
#include "binned.cuh"
#include "open_groups.h"
#include <cfloat>

namespace svoxb {

constexpr int kModeForward = 0;
constexpr int kModeForwardLogged = 2;  // forward that also records its items for the backward

// Floats per record of a colour basis size (0: RGBA).
template <int BD>
struct RecordLength { static constexpr int K = BD == 0 ? 4 : 3 * BD + 1; };

// How a record moves between global memory and its staging row in shared memory: as the
// 16-byte words that cover it.  A record whose length is no multiple of four starts at any
// float, so its row holds up to three floats of its neighbours on either side.
template <int K>
struct RecordShape {
    static constexpr bool ALIGNED = K % 4 == 0;
    static constexpr int WORDS = ALIGNED ? K / 4 : (K + 3 + 3) / 4;
    static constexpr int GROUP = WORDS <= 1 ? 1 : WORDS <= 2 ? 2 : WORDS <= 4 ? 4
                                 : WORDS <= 8 ? 8 : WORDS <= 16 ? 16 : 32;  // lanes per record
    static constexpr int RPP = 32 / GROUP;                                  // records per pass
    // row stride in floats: 16-byte rows, an odd number of 16-byte units (no bank conflicts
    // among the 16-byte reads of different rows)
    static constexpr int STRIDE = 4 * (WORDS | 1);
};

// Item log: what a logged forward leaves behind so that the backward pass can
// replay the contributing samples without marching again and without reading
// the leaf records a second time.  int32 words:
//   [0] chunks asked for   [2] bin shift   [3] number of bins
//   [1] items in units of 32, each warp's rounded up (items alone would outgrow a word)
//   [kLogGivenUp] not 0: the log has holes and must not be replayed, whatever its size
//   [kLogBricks], [.. + 1] counter of an index built in the log's memory (see fallback_index)
//   [kLogNext + p]         units taken of scatter part p, [kLogNext + kMaxParts + p] blocks done
//   [kLogBins + b]         groups of bin b      [kLogCleared + b]  cleared units of bin b
//   [kLogCounts + g]       items of group g (bits 0-7) and its bin (bits 8-)
//   then, 128-byte aligned, 32 packets of 12 words per chunk, and the order of the groups by
//   bin (one word per group; only with several bins).
// A PACKET is one contributing sample: {slot, ray, q0, q1} {q2, h0, h1, h2} {dd, view
// direction}, with q = weight * sg * (1 - sg) per colour channel (sg the channel's sigmoid), h =
// colour * T + S (T the transmittance after the sample, S the ray's colour sum up to and
// including it) and dd = delta_t * delta_scale, times the derivative of the density's softplus
// if that is on.  With g = grad_out[ray] the reference's gradient of the sample is
//   d/d coef  = basis[i] * q * g * (1 + 2 pad)                  (svox/csrc/rt_kernel.cu:386-392)
//   d/d sigma = dd * sum_ch g (h - out[ray])                    (:462-471)
// because its running `accum` after the sample equals <g, out> - <g, S>: every packet is
// self-contained and the backward can take them in any order.
//
// One bin: a GROUP is one chunk, a batch of the forward, in the order of the march.  Several
// bins (ranges of leaf slots): a group is kSortedChunks chunks, and every block keeps an open
// group per bin, so that the backward can take the packets range by range and the gradient
// stays in L2 meanwhile.
constexpr int kMaxParts = 16;   // the scatter can run in up to 16 parts (bin ranges)
constexpr int kLogBricks = 8;
constexpr int kLogNext = 32;
constexpr int kLogBins = kLogNext + 2 * kMaxParts;
constexpr int kLogCleared = kLogBins + kMaxBins;
constexpr int kLogCounts = kLogCleared + kMaxBins;
constexpr int kPacketWords = 12;
constexpr int kLogGrab = 8;        // groups a warp takes at least per bump of the counter ...
constexpr int kSortedGrab = 2;     // ... of a sorted log
__host__ __device__ inline int64_t log_packets_at(int64_t capacity) {
    return (kLogCounts + capacity + 31) & ~(int64_t)31;
}
__host__ __device__ inline int64_t log_order_at(int64_t capacity) {
    return log_packets_at(capacity) + capacity * (32 * kPacketWords);
}
__host__ __device__ inline int64_t log_words(int64_t capacity) {
    return log_order_at(capacity) + capacity + kMaxBins;   // ... and cursors of the ordering
}

// The log as a kernel gets it: written by a logged forward, the gate of a fallback march.
struct LogArgs {
    int32_t* log = nullptr;
    int64_t capacity = 0;
    int shift = 0, n_bins = 1;
};

// The index (tens of MB, re-read hundreds of times per launch) must stay in L2 while the leaf
// records and gradients (GBs, touched a few times each) stream through it.  (Without the hint 300 rays
// with gradient take 354 us instead of 302, 4096 467 instead of 459; calls that fill the device level.)
__device__ __forceinline__ int2 ld_keep(const int2* a, uint64_t pol) {
    int2 v;
    asm volatile("ld.global.nc.L2::cache_hint.v2.s32 {%0, %1}, [%2], %3;"
                 : "=r"(v.x), "=r"(v.y)
                 : "l"(a), "l"(pol));
    return v;
}
// The 64-byte L2 fetch granularity is a measured choice: records are 112-196 bytes at arbitrary
// 16-byte offsets, and the logged forward of the training step runs 1 % faster with it than with the
// default granularity and 6 % faster than with 256 bytes.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, uint64_t pol) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global.L2::cache_hint.L2::64B [%0], [%1], 16, %2;" ::"r"(s),
                 "l"(gmem), "l"(pol)
                 : "memory");
}
// a - b, both halves in one instruction.
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\t"
        "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "sub.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// Adds the 16-byte word `word` of a gradient row to its place.  The row holds the record's K
// floats from offset `off` on, zeros around them; `rec` is the record's first float.  With a
// gradient buffer that is not 16-byte aligned the record's floats go one by one.
template <int K>
__device__ __forceinline__ void flush_word(float* __restrict__ rec, int off, int word,
                                           const float4 x, bool vec_ok, uint64_t pol) {
    if (RecordShape<K>::ALIGNED || vec_ok) {
        red_add_v4_hint(rec - off + 4 * word, x.x, x.y, x.z, x.w, pol);
    } else {
        const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = 4 * word + i - off;
            if (e >= 0 && e < K) atomicAdd(rec + e, v[i]);
        }
    }
}

// Offset of record `slot` from the 16-byte word it starts in, in floats.
template <int K>
__device__ __forceinline__ int record_offset(const float* base, uint32_t slot) {
    if (RecordShape<K>::ALIGNED) return 0;
    return (int)((reinterpret_cast<uintptr_t>(base) >> 2) + slot * (uint32_t)(K & 3)) & 3;
}

// Shared memory of one warp.
template <int BD, int MODE>
struct alignas(16) WarpQueue {
    static constexpr int K = RecordLength<BD>::K;
    static constexpr bool LOG = MODE == kModeForwardLogged;
    using Shape = RecordShape<K>;
    // two batches: items being collected, and what spills over (the batch in flight lies in
    // registers; a queue of 96 items left the SH16 forward 28 KB of L1 instead of 60, 1.10 ms per
    // 800x800 view instead of 1.05)
    static constexpr int CAP = 64;
    // per ray: colour basis and, for the log, the view direction; odd stride: no bank conflicts
    // among different owners (which 16-byte reads of the basis would have)
    static constexpr int RAYW = (BD + (LOG ? 3 : 0)) | 1;
    // An item in words: slot, optical depth (step length * delta_scale * density), owner lane and, for
    // the log, step length * delta_scale.  With the latter it goes as one 16-byte word, else as an
    // 8-byte and a 4-byte one (with 16 bytes the SH16 forward's five blocks would no longer leave
    // 60 KB of L1).  For 25 logged functions the owner is a byte: with more a fourth block would
    // not fit the SM.
    static constexpr bool BYTE = LOG && BD == 25;
    static constexpr bool WIDE = LOG && !BYTE;
    struct Item {
        uint32_t slot;
        float depth, length;
        int owner;
    };
    // Staging rows (cp.async targets).  After lane i has read row i it reuses the
    // row's first words for the item's results.
    alignas(16) float rows[32 * Shape::STRIDE];
    alignas(16) uint32_t items[CAP * (WIDE ? 4 : 3)];
    unsigned char owners[BYTE ? CAP : 1];
    float rayv[32][RAYW];

    __device__ __forceinline__ void put(int i, const Item& x) {
        const uint32_t depth = __float_as_uint(x.depth), length = __float_as_uint(x.length);
        if (WIDE) {
            reinterpret_cast<uint4*>(items)[i] = make_uint4(x.slot, depth, length, x.owner);
        } else {
            reinterpret_cast<uint2*>(items)[i] = make_uint2(x.slot, depth);
            items[2 * CAP + i] = BYTE ? length : x.owner;
            if (BYTE) owners[i] = (unsigned char)x.owner;
        }
    }
    __device__ __forceinline__ Item get(int i) const {
        if (WIDE) {
            const uint4 w = reinterpret_cast<const uint4*>(items)[i];
            return {w.x, __uint_as_float(w.y), __uint_as_float(w.z), (int)w.w};
        }
        const uint2 w = reinterpret_cast<const uint2*>(items)[i];
        const uint32_t v = items[2 * CAP + i];
        return {w.x, __uint_as_float(w.y), BYTE ? __uint_as_float(v) : 0.f, BYTE ? owners[i] : (int)v};
    }
};

// Marks the table cells that the rays pass, at points a quarter of a cell apart: for a few rays
// only these get bricks, instead of the whole scene.  A cell that is clipped between two points
// goes unmarked; the march then walks the tree for its samples there.  One warp per ray.
template <class Source>
__global__ void __launch_bounds__(128)
mark_cells_kernel(TreeArgs tr, Source src, svoxb_render_options opt, int64_t tickets, int L,
                  uint8_t* __restrict__ marks) {
    const int64_t ticket = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int64_t ray = ticket < tickets ? src.pick(ticket) : -1;
    if (ray < 0) return;
    Ray r;
    src.load(ray, tr, opt, r);
    ray_setup(r, tr.scaling);
    if (!r.hit) return;
    const int side = 1 << L;
    const float step = 0.25f / (float)side;
    for (int k = threadIdx.x & 31; k < 8 * side; k += 32) {      // a diagonal is sqrt(3) long
        const float t = r.tmin + (float)k * step;
        if (!(t < r.tmax)) break;
        const int x = (int)(clamp01(r.ox + t * r.dx) * (float)side),
                  y = (int)(clamp01(r.oy + t * r.dy) * (float)side),
                  z = (int)(clamp01(r.oz + t * r.dz) * (float)side);
        marks[(((x << L) + y) << L) + z] = 1;
    }
}

// State of a lane: the samples its ray may still take (marching), or one of these.  (A ray that met a
// damaged node ends like any other, its tmax no number.)
enum { kMarching = 1, kCapped = 0, kNeedRay = -1, kEnded = -2, kExhausted = -3 };

constexpr int kMarchBlock = 128;

// Blocks of kMarchBlock threads per SM the kernel is compiled for: as many as shared memory
// holds, at most 6 (24 warps, 80 registers per thread).  Measured on the logged forward of 2^20
// rays, SH9: 8 blocks (64 registers, no L1 left beside 213 KB of queues) 5.0 ms, 7 blocks 3.6,
// 6 blocks 3.5, 5 blocks 3.7.
constexpr int kMarchBlocks = 6;

// A batch of few rays (march_shape leaves no more than kSpreadWarps warps per SM with work) goes
// through blocks of this size, compiled for 16 warps per SM and thus 128 registers; the march of 4096
// rays of the 512^3 shell, SH9, takes 204 us instead of 237.  The whole call, us, blocks of 128 / of 64
// (512^3 shell, rendering alone; the line is at 75 776 rays):
//            4096 rays   20 000      50 000      75 000      100 000     140 000
//     RGBA   280 / 273   310 / 298   334 / 335   349 / 345   379 / 358   454 / 469
//     SH4    306 / 298   343 / 331   383 / 373   400 / 381   413 / 495   552 / 536
//     SH9    325 / 313   373 / 354   404 / 385   425 / 398   461 / 531   608 / 636
//     SH16   338 / 322   394 / 359   456 / 417   487 / 467   630 / 614   724 / 734
// Beyond the line a warp's 32 lanes all have rays and 16 warps are too few of them; up to it all
// formats gain, images too (224x224 to 272x272 pixels 1 to 2 %).  Logged, with the backward: SH4
// and SH9 7 to 10 % (128^3), SH16 level to 6 %, SH25 level to 2 %, whose kernel has 121 to 128 registers
// either way: there the smaller blocks only share rays out more evenly.
constexpr int kFewBlock = 64;
constexpr int kSpreadWarps = 16;

template <int BD, int MODE>
constexpr int march_blocks_per_sm() {
    const size_t smem = (kMarchBlock / 32) * sizeof(WarpQueue<BD, MODE>) + 1024;
    const int fit = (int)(227 * 1024 / smem);
    return fit > kMarchBlocks ? kMarchBlocks : fit < 1 ? 1 : fit;
}

template <int BD, int MODE>
constexpr int few_blocks_per_sm() {
    const int most = kSpreadWarps / (kFewBlock / 32);
    const int fit = (int)(227 * 1024 / ((kFewBlock / 32) * sizeof(WarpQueue<BD, MODE>) + 1024));
    return fit < most ? fit : most;
}

// A forward that sorts its log into bins runs as one block per SM, so that a bin has one open
// group per SM and the lines being filled stay in L2 until they are full.
constexpr size_t bin_smem(int n_bins) {
    return (size_t)n_bins * (sizeof(uint32_t) + kOpenGroups * sizeof(uint64_t));
}
constexpr size_t kBinSmem = bin_smem(kMaxBins);
template <int BD>
constexpr int sorted_march_block() {
    // If it costs no more than a warp, within 196 KB with half of the bins, the next smaller split of an
    // SM's memory, which leaves 60 KB of L1 instead of 28 (SH16 with 62 bins: 19 warps instead of 20,
    // logged 800x800 view 1.26 -> 1.21 ms; SH25 stays at 15 warps, 13 took 417 us instead of 387 for a
    // 640x640 view).
    constexpr size_t one = sizeof(WarpQueue<BD, kModeForwardLogged>);
    const int warps = 4 * march_blocks_per_sm<BD, kModeForwardLogged>();
    int most = (int)((227 * 1024 - 1024 - kBinSmem) / one);
    const int fit = (int)((196 * 1024 - 1024 - kBinSmem / 2) / one);
    if (most > warps) most = warps;
    return 32 * (fit < most - 1 ? most : fit < most ? fit : most);
}

// clamp01's upper bound
constexpr float kPosMax = (float)(1.0 - 1e-6);

// The march clamps positions with a saturating FMA, which maps NaN to 0 where clamp01 gives its
// upper bound, and leaves out _dda_unit's bound of 1e9 on the exit distance, which matters
// without a direction only.  So a NaN origin is replaced by one beyond the upper bound, and a
// ray without a direction, for which the reference takes one sample at the cube's upper corner,
// is given a position and an extent that make the march do just that.
__device__ __forceinline__ void march_ready(Ray& r) {
    if (r.ox != r.ox) { r.ox = 1.f; r.dx = r.dx == r.dx ? 0.f : r.dx; }
    if (r.oy != r.oy) { r.oy = 1.f; r.dy = r.dy == r.dy ? 0.f : r.dy; }
    if (r.oz != r.oz) { r.oz = 1.f; r.dz = r.dz == r.dz ? 0.f : r.dz; }
    if (r.dx == r.dx && r.dy == r.dy && r.dz == r.dz) return;
    r.ox = r.oy = r.oz = 1.f;
    r.dx = r.dy = r.dz = 0.f;
    r.ix = r.iy = r.iz = 1.f;
    r.tmax = __int_as_float(__float_as_int(r.tmin) + 1);
}

// How a launch deals out its rays: lanes of a warp that take rays, log2 of the tickets a block
// draws in a row, and how many lanes of a warp must be without a ray before they refill.
struct MarchShape {
    int lanes, granule_shift, refill;
};

template <int BD, int MODE, int BLOCK, class Source>
__global__ void
__launch_bounds__(BLOCK, BLOCK == kMarchBlock ? march_blocks_per_sm<BD, MODE>()
                         : BLOCK == kFewBlock ? few_blocks_per_sm<BD, MODE>() : 1)
render_queue_kernel(TreeArgs tr, Source src, svoxb_render_options opt, TreeIndex index,
                    int64_t tickets, float* __restrict__ out, LogArgs lg, MarchShape shape) {
    constexpr int K = RecordLength<BD>::K;
    constexpr bool LOG = MODE == kModeForwardLogged;
    using WQ = WarpQueue<BD, MODE>;
    using Shape = RecordShape<K>;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ unsigned s_next;
    if (threadIdx.x == 0) s_next = 0;
    // sorted log: items this block has put into each bin, and its last groups of the bin
    constexpr bool SORTED = LOG && BLOCK > kMarchBlock;
    uint64_t* s_open = reinterpret_cast<uint64_t*>(s_raw + (BLOCK / 32) * sizeof(WQ));
    uint32_t* s_count = reinterpret_cast<uint32_t*>(s_open + lg.n_bins * kOpenGroups);
    if (SORTED) {
        for (int i = threadIdx.x; i < lg.n_bins * kOpenGroups; i += BLOCK) s_open[i] = 0;
        for (int i = threadIdx.x; i < lg.n_bins; i += BLOCK) s_count[i] = 0;
    }
    if (LOG && blockIdx.x == 0 && threadIdx.x == 0) {
        lg.log[2] = lg.shift;
        lg.log[3] = lg.n_bins;
    }
    // Kept in registers: left to itself the compiler works these three out again at every use.
    int lane = threadIdx.x & 31;
    uint32_t queue = (uint32_t)__cvta_generic_to_shared(s_raw) + (threadIdx.x >> 5) * (uint32_t)sizeof(WQ);
    unsigned below = (1u << lane) - 1u;
    asm volatile("" : "+r"(lane), "+r"(queue), "+r"(below));
    WQ& q = *reinterpret_cast<WQ*>(__cvta_shared_to_generic(queue));
    const uint64_t pol_stream = l2_policy_stream(), pol_keep = l2_policy_keep();
    __syncthreads();
    const float d_rgb_pad = 1 + 2 * opt.rgb_padding;
    const float bg = opt.background_brightness;
    // Items are evaluated 32 at a time, where all lanes have one, and folded into the ray in order;
    // there it is decided whether the ray stops early, and the march is told.  Before that it ends a
    // ray once its summed optical depth is beyond that of the threshold by more than the
    // roundings of 2^16 factors can amount to (only where no density is negative, which would make the
    // two part further, and where the product does not run into denormal numbers before the
    // threshold).  What it takes behind the stop counts for nothing, a damaged node there and the sample
    // cap too.
    const bool early = MODE == kModeForward && opt.stop_thresh > 0.f;
    float deep = __int_as_float(0x7f800000);
    if (early && opt.sigma_thresh >= 0.f && opt.stop_thresh >= FLT_MIN) {
        deep = -logf(opt.stop_thresh);
        deep += 0.0625f + fmaxf(deep, 0.f) * 0.015625f;
    }

    // ---- per-lane state -------------------------------------------------------
    Ray r{};        // (lanes without a ray look up entries too)
    int64_t ray = 0;
    int state = lane < shape.lanes ? kNeedRay : kExhausted;
    // max(1 / direction, 0), where registers allow (1 % of an image's march)
    constexpr bool MAXES = MODE == kModeForward;
    float mx = 0.f, my = 0.f, mz = 0.f;
    float t = 0.f, light = 1.f;          // transmittance after the items folded
    float depth = 0.f;                   // optical depth of the items pushed
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;  // colour sums
    bool stopped = false;
    uint32_t cur_cell = 0xffffffffu;   // table cell of the brick used last ...
    uint32_t cur_brick = 0;            // ... and where the brick lies in the index
    // cursor: the position of the lane's next sample, and the index words requested for it
    float px = 0.f, py = 0.f, pz = 0.f;
    int2 entry = make_int2(0, 0);
    uint32_t cell = 0;                 // ... and its table cell
    // queue: ring of two batches; `qn` items collected from ring position `head` on
    int head = 0, qn = 0;
    // my items, the first in the highest bit: first 32, spilled, in flight
    unsigned mine = 0u, mine_next = 0u, mine_fly = 0u;
    int fly = 0;                       // items in flight, and this lane's
    typename WQ::Item fly_item{0u, 0.f, 0.f, 0};
    // logged forward: groups the warp has taken from the log but not used, items written
    int log_group = 0, log_left = 0, log_items = 0;

    // Places the cursor at parameter t and requests the index words there, to be consumed one
    // iteration later: the brick's, if the ray is still in the table cell whose brick it used
    // last, else the table's.
    auto place_cursor = [&]() {
        px = fminf(__saturatef(mad_site<FC_POS>(t, r.dx, r.ox)), kPosMax);
        py = fminf(__saturatef(mad_site<FC_POS>(t, r.dy, r.oy)), kPosMax);
        pz = fminf(__saturatef(mad_site<FC_POS>(t, r.dz, r.oz)), kPosMax);
    };
    auto request_words = [&]() {
        // the sums' low bits: the position in cells of a brick, exactly
        const float2 xy = __fadd2_rz(make_float2(px, py), make_float2(index.fine, index.fine));
        const uint32_t ux = __float_as_uint(xy.x), uy = __float_as_uint(xy.y),
                       uz = __float_as_uint(__fadd_rz(pz, index.fine));
        // places in bytes: an entry has 2^kBrickLevels of them
        cell = ((ux & index.cell_mask) * index.row + (uy & index.cell_mask)) * index.row +
               (uz & index.cell_mask);
        const uint32_t c = ((ux & 7u) << 9) | ((uy & 7u) << 6) | ((uz & 7u) << 3);
        const uint32_t at = cell == cur_cell ? cur_brick + c : cell;
        entry = ld_keep(reinterpret_cast<const int2*>(reinterpret_cast<const char*>(index.table) + at), pol_keep);
    };

    // Takes the first n (<= 32) collected items as the batch in flight and requests their
    // records: consecutive lanes copy consecutive 16-byte words, asynchronously.
    auto request = [&](int n) {
        fly_item = q.get(head + lane);
        const uint32_t slot = fly_item.slot;
        mine_fly = mine;
        mine = mine_next;
        mine_next = 0u;
        fly = n;
        head ^= 32;
        qn = qn > 32 ? qn - 32 : 0;
        int l = lane;
        asm volatile("" : "+r"(l));
        const int sub = l / Shape::GROUP, w = l % Shape::GROUP;
        const float* base = tr.data + 4 * w;
        float* row = q.rows + sub * Shape::STRIDE + 4 * w;
#pragma unroll
        for (int p = 0; p < Shape::GROUP; ++p) {
            const uint32_t s = __shfl_sync(0xffffffffu, slot, p * Shape::RPP + sub);
            if (p * Shape::RPP + sub < n && w < Shape::WORDS) {
                const float* rec = base + (size_t)s * K;
                if (!Shape::ALIGNED)
                    rec = reinterpret_cast<const float*>(reinterpret_cast<uintptr_t>(rec) &
                                                         ~(uintptr_t)15);
                cp_async16(row + p * Shape::RPP * Shape::STRIDE, rec, pol_stream);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        __syncwarp();        // the items' places are free again
    };

    // Waits for the records of the batch in flight and evaluates it.
    auto evaluate = [&]() {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const int nb = fly;
        const bool active = lane < nb;
        const uint32_t b_slot = fly_item.slot;
        float* row = q.rows + lane * Shape::STRIDE;
        const int off = record_offset<K>(tr.data, b_slot);
        const int own = fly_item.owner & 31;
        // (a lane without an item computes along on what its row and place held before)
        float sg[3], col[3], raw_sigma = 0.f;
        const float att = expf(-fly_item.depth);
        {
            float tmp[3] = {0.f, 0.f, 0.f};
            const float* ray_basis = q.rayv[own];
            if (BD == 0) {
                const float4 x = *reinterpret_cast<const float4*>(row);
                tmp[0] = x.x; tmp[1] = x.y; tmp[2] = x.z;
                raw_sigma = x.w;
            } else if (Shape::ALIGNED) {
                constexpr int B = BD > 0 ? BD : 1;
                float bs[B];
#pragma unroll
                for (int i = 0; i < B; ++i) bs[i] = ray_basis[i];
#pragma unroll
                for (int w = 0; w < K / 4; ++w) {
                    const float4 x = reinterpret_cast<const float4*>(row)[w];
                    const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int e = 4 * w + i;
                        if (e < K - 1) tmp[e / B] = __fmaf_rn(bs[e % B], v[i], tmp[e / B]);
                        else raw_sigma = v[i];
                    }
                }
            } else {
                // The row's 16-byte words as they are: float j of the row is coefficient j - off,
                // so basis function (j - off) mod BD takes it, which is one register for all
                // three channels; only the first three of a channel's places depend on `off`.  (A
                // 49-float record as single floats met three bank conflicts a read: 1.03 ms per
                // 800x800 view instead of 1.01.)
                constexpr int B = BD > 0 ? BD : 1;
                float bs[B];
#pragma unroll
                for (int m = 0; m < B; ++m)
                    bs[m] = ray_basis[m >= 3 || m >= off ? m - off : m - off + B];
#pragma unroll
                for (int w = 0; w < Shape::WORDS; ++w) {
                    const float4 x = reinterpret_cast<const float4*>(row)[w];
                    const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int j = 4 * w + i, m = j % B, c = j / B;
                        if (m >= 3 || m >= off) {
                            if (c < 3) tmp[c < 3 ? c : 0] = __fmaf_rn(bs[m], v[i], tmp[c < 3 ? c : 0]);
                            else if (m == off) raw_sigma = v[i];
                        } else if (c > 0) {
                            tmp[c > 0 ? c - 1 : 0] = __fmaf_rn(bs[m], v[i], tmp[c > 0 ? c - 1 : 0]);
                        }
                    }
                }
            }
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                sg[ch] = sigmoid_ref(tmp[ch]);
                col[ch] = sg[ch] * d_rgb_pad - opt.rgb_padding;
            }
            *reinterpret_cast<float4*>(row) = make_float4(col[0], col[1], col[2], att);
        }
        __syncwarp();
        // every owner folds in its items, in march order
        for (unsigned m = mine_fly; m != 0u;) {
            const int first = __clz(m);
            m &= ~(0x80000000u >> first);
            float4* res = reinterpret_cast<float4*>(q.rows + first * Shape::STRIDE);
            const float4 x = *res;
            // res->w: the transmittance before the item, 0 where the ray has stopped
            const float before = stopped ? 0.f : light;
            const float weight = before * (1.f - x.w);
            if (!stopped) {
                a0 = __fmaf_rn(weight, x.x, a0);
                a1 = __fmaf_rn(weight, x.y, a1);
                a2 = __fmaf_rn(weight, x.z, a2);
                light = light * x.w;
                stopped = light <= opt.stop_thresh;
            }
            if (LOG) *res = make_float4(a0, a1, a2, before);
            else res->w = before;
        }
        mine_fly = 0u;
        fly = 0;
        if (early && stopped && state >= kMarching) state = kEnded;
        __syncwarp();
        // (nothing of an item that its ray did not reach, whatever its density)
        if (tr.weight_accum != nullptr && active && row[3] != 0.f)
            accumulate_weight(tr, b_slot, row[3] * (1.f - att));
        if (LOG) {
            int32_t* log = lg.log;                   // (computed from here, not kept)
            int64_t capacity = lg.capacity;
            asm volatile("" : "+l"(log), "+l"(capacity));
            const int log_limit = SORTED ? (int)(capacity / kSortedChunks) : (int)capacity;
            int32_t* const log_counts = log + kLogCounts;
            int4* const packets = reinterpret_cast<int4*>(log + log_packets_at(capacity));
            // lane i writes the packet of item i, now that its ray's colour sums are known: to
            // place i of the batch's chunk, or to the next place of its bin
            const int ray_id = __shfl_sync(0xffffffffu, (int)ray, own);
            int bin = 0, place = lane;
            uint32_t number = 0;
            if (SORTED && active) {
                bin = (int)(b_slot >> lg.shift);
                const uint32_t n = atomicAdd(&s_count[bin], 1u);
                place = (int)(n % kSortedItems);
                number = n / kSortedItems;
            }
            // lanes that open a group: the first of its items
            const bool opens = SORTED ? active && place == 0 : lane == 0;
            const unsigned opening = __ballot_sync(0xffffffffu, opens);
            const int n_open = __popc(opening);
            const int mine_open = __popc(opening & below);
            int group_id = log_group + mine_open;
            if (n_open > log_left) {
                constexpr int GRAB = SORTED ? kSortedGrab : kLogGrab;
                constexpr int UNIT = SORTED ? kSortedChunks : 1;
                const int more = n_open - log_left > GRAB ? n_open - log_left : GRAB;
                int c = 0;
                if (lane == 0) c = atomicAdd(log, more * UNIT) / UNIT;
                c = __shfl_sync(0xffffffffu, c, 0);
                if (mine_open >= log_left) group_id = c + mine_open - log_left;
                log_group = c + n_open - log_left;
                log_left += more - n_open;
            } else {
                log_group += n_open;
                log_left -= n_open;
            }
            if (opens && group_id < log_limit)
                log_counts[group_id] = SORTED ? kSortedItems | (bin << 8) : nb;
            if (SORTED) {
                volatile uint64_t* open = s_open + bin * kOpenGroups + open_group_place(number);
                if (opens) *open = open_group_entry(number, group_id);
                __syncwarp();
                if (active && !opens) {
                    // another warp may be about to publish the group's id
                    uint64_t v = *open;
                    int tries = 0;
                    while (!open_group_is(v, number) && ++tries < (1 << 14)) {
                        __nanosleep(32);
                        v = *open;
                    }
                    group_id = open_group_id(v);
                    if (!open_group_is(v, number)) {    // never seen: give the log up, march instead
                        log[kLogGivenUp] = 1;
                        group_id = 0x7fffffff;
                    }
                }
                __syncwarp();
            } else {
                group_id = __shfl_sync(0xffffffffu, group_id, 0);
            }
            if (active && group_id < log_limit) {
                const float4 sums = *reinterpret_cast<const float4*>(row);
                const float b_w = sums.w * (1.f - att), b_T = sums.w * att;
                // the step length carries d softplus / d raw density, the one factor the
                // density gradient needs from the raw value (svox/csrc/rt_kernel.cu:469-470)
                float b_dd = fly_item.length;
                if (opt.density_softplus) b_dd *= sigmoid_ref(raw_sigma - 1);
                int qf[3];
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) {
                    // w sg (1 - sg), the product with 1 - sg rounded once
                    const float part = b_w * sg[ch];
                    qf[ch] = __float_as_int(__fmaf_rn(-part, sg[ch], part));
                }
                const float* vd = &q.rayv[own][BD];
                int4* to = packets + ((int64_t)group_id * (SORTED ? kSortedItems : 32) + place) *
                                         (kPacketWords / 4);
                const uint64_t pol = SORTED ? l2_policy_keep() : pol_stream;
                st_hint16(to, make_int4((int)b_slot, ray_id, qf[0], qf[1]), pol);
                st_hint16(to + 1, make_int4(qf[2], __float_as_int(__fmaf_rn(col[0], b_T, sums.x)),
                                            __float_as_int(__fmaf_rn(col[1], b_T, sums.y)),
                                            __float_as_int(__fmaf_rn(col[2], b_T, sums.z))), pol);
                st_hint16(to + 2, make_int4(__float_as_int(b_dd), __float_as_int(vd[0]),
                                            __float_as_int(vd[1]), __float_as_int(vd[2])), pol);
            }
            log_items += nb;
            __syncwarp();
        }
    };

    // marching lanes at which the others are refilled: at none at the latest
    auto refill_line = [&]() {
        const int alive = __popc(__ballot_sync(0xffffffffu, state != kExhausted));
        return alive > shape.refill ? alive - shape.refill : 0;
    };
    int refill_at = refill_line();
    for (;;) {
        // ---- lanes that are not marching: finish, refill, termination ---------------------
        int marching_lanes = __popc(__ballot_sync(0xffffffffu, state >= kMarching));
        if (marching_lanes <= refill_at) {
            if (__any_sync(0xffffffffu, state < kMarching && (mine | mine_next | mine_fly) != 0u)) {
                __syncwarp();
                while (fly > 0 || qn > 0) {
                    if (fly > 0) evaluate();
                    if (qn > 0) request(qn < 32 ? qn : 32);
                }
            }
            if (state == kEnded || state == kCapped) {
                const int fault = state == kCapped ? SVOXB_ERR_MARCH
                                  : r.tmax != r.tmax ? SVOXB_ERR_TREE : 0;
                if (fault != 0 && !(early && stopped)) report(fault);
                state = kNeedRay;
                if (stopped) {
                    const float scale = 1.0 / (1.0 - light);
                    out[3 * ray + 0] = a0 * scale;
                    out[3 * ray + 1] = a1 * scale;
                    out[3 * ray + 2] = a2 * scale;
                } else {
                    out[3 * ray + 0] = a0 + light * bg;
                    out[3 * ray + 1] = a1 + light * bg;
                    out[3 * ray + 2] = a2 + light * bg;
                }
            }
            if (state == kNeedRay) {
                // What a ray's set-up derives from the call's arguments is not to be kept in registers
                // through the march.
                Source rays = src;
                TreeArgs tree = tr;
                svoxb_render_options how = opt;
                rays.pin();
                asm volatile("" : "+l"(tree.offset), "+l"(tree.scaling), "+l"(tree.extra));
                asm volatile("" : "+r"(how.ndc_width), "+r"(how.ndc_height), "+f"(how.ndc_focal),
                                  "+r"(how.min_comp), "+r"(how.max_comp));
                const unsigned ticket = atomicAdd(&s_next, 1u);
                const int gs = shape.granule_shift;
                const int64_t first =
                    ((int64_t)blockIdx.x + (int64_t)gridDim.x * (ticket >> gs)) << gs;
                const int64_t turn = first + (ticket & ((1u << gs) - 1u));
                if (first >= tickets) {
                    state = kExhausted;
                } else if (turn < tickets && (ray = rays.pick(turn)) >= 0) {
                    rays.load(ray, tree, how, r);
                    ray_setup(r, tree.scaling);
                    if (!r.hit || !(r.tmin < r.tmax)) {
                        out[3 * ray + 0] = bg; out[3 * ray + 1] = bg; out[3 * ray + 2] = bg;
                    } else {
                        march_ready(r);
                        state = kMaxSteps;
                        t = r.tmin; light = 1.f; depth = 0.f; stopped = false;
                        mx = fmaxf(r.ix, 0.f); my = fmaxf(r.iy, 0.f); mz = fmaxf(r.iz, 0.f);
                        place_cursor();
                        request_words();
                        if (BD > 0) {
                            float basis[BD > 0 ? BD : 1];
                            colour_basis<(BD > 0 ? BD : 1), Source::kLobes>(tree, how, r.vdir, basis);
#pragma unroll
                            for (int i = 0; i < BD; ++i)
                                q.rayv[lane][i] =
                                    (i < how.min_comp || i > how.max_comp) ? 0.f : basis[i];
                        }
                        if (LOG) {
#pragma unroll
                            for (int i = 0; i < 3; ++i) q.rayv[lane][BD + i] = r.vdir[i];
                        }
                        a0 = a1 = a2 = 0.f;
                    }
                }
            }
            __syncwarp();
            refill_at = refill_line();
            if (!__any_sync(0xffffffffu, state >= kMarching)) {
                if (!__any_sync(0xffffffffu, state != kExhausted)) break;
                continue;
            }
        }

        // ---- G step: every lane consumes the words requested one iteration ago --------------
        // (without branches but for the rare cases: lanes that have nothing to do compute along)
        const bool to_brick = entry.x < 0;
        if (to_brick) {
            // the table cell has a brick: the sample is looked up there
            cur_cell = cell;
            cur_brick = (index.bricks + (uint32_t)entry.x * kBrickCells) * 8;    // (drops the sign)
        }
        const bool on = state >= kMarching && !to_brick;
        uint32_t slot = (uint32_t)entry.y & 0x0fffffffu;
        float sigma = __int_as_float(entry.x);
        bool item = on && entry.x <= kWordInf;      // the leaf passes the density test
        // side of the leaf's cube, 2^-depth
        float inv_cube = __int_as_float((127 << 23) - (int)((uint32_t)entry.y >> 28 << 23));
        // Lower corner of the leaf: a number whose last place is the leaf's side takes in the
        // position's multiples of it and drops the rest.
        float coarse = __int_as_float(__float_as_int(inv_cube) + (kPosBits << 23));
        const float2 pxy = make_float2(px, py), coarse2 = make_float2(coarse, coarse);
        float2 cxy = sub2(__fadd2_rz(pxy, coarse2), coarse2);
        float cz = __fsub_rn(__fadd_rz(pz, coarse), coarse);
        const bool rare = on && entry.x >= kWordFetch;
        if (__any_sync(0xffffffffu, rare)) {
            // seldom: a tree deeper than the index, a density that is not in the word
            if (rare) {
                float raw = 0.f;
                if (entry.x == kWordWalk) {
                    const float big = (float)(1 << 24);
                    const int level = (int)((uint32_t)entry.y >> 28);
                    const int ix = (int)(px * big), iy = (int)(py * big), iz = (int)(pz * big);
                    const Walked f = walk_to_leaf(tr.child, tr.data, K, tr.M,
                                                  level > index.level ? (int64_t)slot : 0,
                                                  level > index.level ? level - 1 : 0, ix, iy, iz);
                    if (!f.ok) r.tmax = __int_as_float(0x7fffffff);     // ends the ray
                    slot = f.slot;
                    inv_cube = __int_as_float((127 - (f.ok ? f.depth : 1)) << 23);
                    raw = f.raw;
                    coarse = __int_as_float(__float_as_int(inv_cube) + (kPosBits << 23));
                    cxy.x = __fsub_rn(__fadd_rz(px, coarse), coarse);
                    cxy.y = __fsub_rn(__fadd_rz(py, coarse), coarse);
                    cz = __fsub_rn(__fadd_rz(pz, coarse), coarse);
                    // 2^-24 leaves: a float resolves them below 1/2, where the sums would not
                    if (f.ok && f.depth > kPosBits) {
                        cxy.x = (float)ix * (1.f / big);
                        cxy.y = (float)iy * (1.f / big);
                        cz = (float)iz * (1.f / big);
                    }
                } else {
                    raw = __ldg(tr.data + (size_t)slot * K + (K - 1));
                }
                sigma = opt.density_softplus ? softplus_m1(raw) : raw;
                item = r.tmax == r.tmax && sigma > opt.sigma_thresh;
            }
        }
        // Exit distance of the leaf (_dda_unit, svox/csrc/rt_kernel.cu:203-220, in the leaf's own
        // scale).  The point lies inside, so the entry distance is 0 and per axis the larger of
        // t1 = -f*inv and t1 + inv is t1 + max(inv, 0); powers of two commute with rounding, so
        // everything can be done at the tree's scale.
        const float2 exy = __ffma2_rn(MAXES ? make_float2(mx, my)
                                            : make_float2(fmaxf(r.ix, 0.f), fmaxf(r.iy, 0.f)),
                                      make_float2(inv_cube, inv_cube),
                                      __fmul2_rn(sub2(cxy, pxy), make_float2(r.ix, r.iy)));
        const float ez = __fmaf_rn(MAXES ? mz : fmaxf(r.iz, 0.f), inv_cube,
                                   __fmul_rn(__fsub_rn(cz, pz), r.iz));
        const float delta_t = __fadd_rn(fminf(exy.x, fminf(exy.y, ez)), opt.step_size);
        const float length = __fmul_rn(delta_t, r.delta_scale);
        const float thick = __fmul_rn(length, sigma);
        // The same twice: branches here cost long records registers and time, their absence short
        // ones instructions (800x800 view, us, with / without: SH4 772 / 794, SH9 with thresholds 674 /
        // 669, SH16 1054 / 1041, SH25 1328 / 1221; 65536 RGBA rays with gradient 213 / 216).
        if constexpr (BD >= 9) {
            const float next_t = __fadd_rn(t, delta_t);
            bool end = !(next_t < r.tmax);
            if (MODE == kModeForward) {
                depth += item ? thick : 0.f;
                end |= item & (depth > deep);
            }
            t = on ? next_t : t;
            state = on ? (end ? kEnded : state - 1) : state;
        } else if (on) {
            t = __fadd_rn(t, delta_t);
            --state;
            if (MODE == kModeForward && item) depth += thick;
            if (!(t < r.tmax) || (MODE == kModeForward && item && depth > deep))
                state = kEnded;
        }
        place_cursor();
        // (lanes without a ray load along, which saves a branch: 1 to 2 % of a view; not beside the 28 KB
        // of L1 that 25 functions leave: 100 000 such rays 778 us, 721 without)
        if (BD != 25 || state >= kMarching) request_words();

        // ---- push items --------------------------------------------------------------
        const unsigned pushed = __ballot_sync(0xffffffffu, item);
        if (pushed != 0u) {
            const int n = qn + __popc(pushed & below);
            if (item) {
                q.put((head + n) & (WQ::CAP - 1),
                      typename WQ::Item{slot, thick, length, lane});
                const unsigned bit = 0x80000000u >> (n & 31);
                if (n < 32) mine |= bit;
                else mine_next |= bit;
            }
            qn += __popc(pushed);
            if (qn >= 32) {
                __syncwarp();
                if (fly > 0) evaluate();
                request(32);
            }
        }
    }
    if (LOG) {
        const int log_limit = SORTED ? (int)(lg.capacity / kSortedChunks) : (int)lg.capacity;
        int32_t* const log_counts = lg.log + kLogCounts;
        // groups taken but not used hold no items; the last group of a bin holds what it got
        for (int i = lane; i < log_left; i += 32)
            if (log_group + i < log_limit) log_counts[log_group + i] = 0;
        if (lane == 0 && log_items > 0) atomicAdd(lg.log + 1, (log_items + 31) >> 5);
        if (SORTED) {
            __syncthreads();
            for (int b = threadIdx.x; b < lg.n_bins; b += BLOCK) {
                const uint32_t n = s_count[b];
                if (n == 0) continue;
                const uint32_t last = (n - 1) / kSortedItems;
                const uint64_t v = s_open[b * kOpenGroups + open_group_place(last)];
                const int g = open_group_id(v);
                if (!open_group_is(v, last)) lg.log[kLogGivenUp] = 1;   // overwritten by a late warp
                else if (g < log_limit) log_counts[g] = (int)(n - kSortedItems * last) | (b << 8);
                atomicAdd(lg.log + kLogBins + b, (int)last + 1);
            }
        }
    }
}

}  // namespace svoxb
