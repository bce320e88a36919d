// Backward pass by replay of the forward's item log (see render_queue.cuh for the packets).
//
// The logged forward has already found every contributing sample, evaluated its colour sigmoids
// and recorded the ray's colour sums, so the backward neither marches nor reads a leaf record:
// what is left is adding one K-float record per packet into `grad_data`.
//
//   scatter  a warp takes packets 32 at a time: lane i reads packet i, forms the colour
//            factors and the density gradient with the ray's grad_out and out, expands them to
//            the K-float record in a shared-memory row; groups of lanes flush the rows with
//            red.global.add.v4.f32.
//
// Where every leaf is touched several times by rays far apart in time, each touch would miss L2
// and cost a read and a write of DRAM (20 GB for 2^20 rays of the 512^3 shell scene, 4.5 ms
// against 1.87 with the clearing, see below).  There the forward sorts its packets into BINS, ranges
// of leaf slots whose gradient spans some tens of MB, and `order` lists the groups of packets bin by
// bin: all SMs work on the same few bins at a time.  The kernel then also clears the gradient, one bin ahead
// of the scatter: the zeros are still in L2 when the packets are added, so a gradient line is
// written to DRAM once and never read (clearing first costs another write, and a read of every
// line touched).  Bound then: L2 atomics, 4.5 sectors per 112-byte record.
#pragma once

#include "render_queue.cuh"

namespace svoxb {

constexpr int kScatterBlock = 256;
constexpr int kScatterBatches = 8;   // batches of 32 packets a warp takes at a time at most
constexpr int kOrderTile = 1024;     // groups a block of the order kernel takes at a time

// First bin of part p when n_bins bins are cut into n_parts ranges.
__host__ __device__ inline int replay_part_first_bin(int p, int n_parts, int n_bins) {
    return (int)(((int64_t)p * n_bins) / n_parts);
}

// Lists the groups of a sorted log bin by bin, with their items in the upper 8 bits (there are fewer
// than 2^24 groups).  `cursor`: kMaxBins zeroed words.
__global__ void __launch_bounds__(256)
order_groups_kernel(int32_t* __restrict__ log, int64_t capacity, int32_t* __restrict__ cursor) {
    __shared__ int s_first[kMaxBins], s_count[kMaxBins];
    if (!log_complete(log, capacity)) return;    // never replayed
    const int n = log[0] / kSortedChunks;
    const int n_bins = log[3] > kMaxBins ? kMaxBins : log[3];
    const int32_t* __restrict__ counts = log + kLogCounts;
    int32_t* __restrict__ order = log + log_order_at(capacity);
    if (threadIdx.x < kMaxBins) {
        int first = 0;
        for (int b = 0; b < (int)threadIdx.x && b < n_bins; ++b) first += log[kLogBins + b];
        s_first[threadIdx.x] = first;
    }
    for (int64_t tile = blockIdx.x; tile * kOrderTile < n; tile += gridDim.x) {
        __syncthreads();
        if (threadIdx.x < kMaxBins) s_count[threadIdx.x] = 0;
        __syncthreads();
        int bin[kOrderTile / 256], rank[kOrderTile / 256], items[kOrderTile / 256];
#pragma unroll
        for (int j = 0; j < kOrderTile / 256; ++j) {
            const int64_t g = tile * kOrderTile + 256 * j + threadIdx.x;
            const int32_t w = g < n ? counts[g] : 0;
            items[j] = w & 0xff;
            bin[j] = items[j] != 0 ? w >> 8 : -1;            // groups without items are left out
            rank[j] = bin[j] >= 0 ? atomicAdd(&s_count[bin[j]], 1) : 0;
        }
        __syncthreads();
        if (threadIdx.x < n_bins && s_count[threadIdx.x] > 0)
            s_count[threadIdx.x] = s_first[threadIdx.x] +
                                   atomicAdd(cursor + threadIdx.x, s_count[threadIdx.x]);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kOrderTile / 256; ++j)
            if (bin[j] >= 0)
                order[s_count[bin[j]] + rank[j]] =
                    (int)((uint32_t)(tile * kOrderTile + 256 * j + threadIdx.x) |
                          (uint32_t)items[j] << 24);
    }
}

template <int K>
struct alignas(16) ScatterSmem {
    using Shape = RecordShape<K>;
    alignas(16) float rows[32 * Shape::STRIDE];
};

// What a scatter adds into.  HESS kernels: the Gauss-Newton diagonal of the squared error (the
// square of each output's derivative summed over the three outputs,
// svox/csrc/rt_kernel.cu:596-605, 683-698), and the gradient too if `grad` is given.
struct ScatterOut {
    float* grad;
    float* hess;
    const float* grad_out;
    const float* fwd_out;
    // sorted log only: leaf slots of the outputs, which the kernel then clears itself, every
    // bin just before it is scattered into; 0: they come cleared
    int64_t zero_slots;
};

template <int BD, int BLOCK, bool HESS, bool LOBES>
__global__ void __launch_bounds__(BLOCK)
replay_scatter_kernel(TreeArgs tr, svoxb_render_options opt, int32_t* __restrict__ log,
                      int64_t capacity, ScatterOut to, int part, int n_parts) {
    constexpr int K = RecordLength<BD>::K;
    using Shape = RecordShape<K>;
    using SM = ScatterSmem<K>;
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int lane = threadIdx.x & 31;
    SM& sm = *reinterpret_cast<SM*>(s_raw + (size_t)(threadIdx.x >> 5) * sizeof(SM));
    const uint64_t pol_keep = l2_policy_keep();
    const float d_rgb_pad = 1 + 2 * opt.rgb_padding;
    constexpr int WARPS = BLOCK / 32;
    __shared__ UnitShared s_units;
    const bool useless = !log_complete(log, capacity);    // then no packet counts
    const int n_bins = log[3] > kMaxBins ? kMaxBins : log[3];
    const bool sorted = n_bins > 1;
    const int lo_bin = sorted ? replay_part_first_bin(part, n_parts, n_bins) : 0,
              hi_bin = sorted ? replay_part_first_bin(part + 1, n_parts, n_bins) : 1;
    // batches of 32 packets a warp takes per unit, and per group
    const int chunks = useless || (!sorted && part != 0) ? 0 : log[0];
    const int share = chunks / ((int)gridDim.x * WARPS * (sorted ? n_bins : 4));
    const int per_group = sorted ? kSortedChunks : 1;
    const int per_warp = share < 1 ? 1 : share > kScatterBatches ? kScatterBatches : share;
    const int32_t* __restrict__ counts = log + kLogCounts;
    const int32_t* __restrict__ order = log + log_order_at(capacity);
    const int4* __restrict__ packets =
        reinterpret_cast<const int4*>(log + log_packets_at(capacity));
    int groups_before = 0;
    for (int b = 0; b < lo_bin && !useless; ++b) groups_before += log[kLogBins + b];
    const UnitCounters counters{log + kLogNext + part, log + kLogNext + kMaxParts + part,
                                log + kLogCleared};
    auto count = [&](int b) { return useless ? 0 : sorted ? log[kLogBins + b] : chunks; };
    auto clear = [&](int64_t from, int64_t until) {
        const int4 none = make_int4(0, 0, 0, 0);
        for (int64_t i = from + 4 * threadIdx.x; i < until; i += 4 * BLOCK) {
            if (!HESS || to.grad != nullptr) st_hint16(to.grad + i, none, pol_keep);
            if (HESS) st_hint16(to.hess + i, none, pol_keep);
        }
    };
    auto work = [&](int first, int end) {
        // lane j: first packet and length of the warp's batch j
        int64_t at = 0;
        int len = 0;
        {
            const int batch = (threadIdx.x >> 5) * per_warp + lane;
            const int i = first + batch / per_group;
            if (lane < per_warp && i < end) {
                const uint32_t g =
                    sorted ? (uint32_t)__ldg(order + i) : (uint32_t)__ldg(counts + i) << 24;
                const int sub = batch % per_group;
                at = ((int64_t)(sorted ? g & 0xffffffu : (uint32_t)i) * per_group + sub) * 32;
                len = (int)(g >> 24) - 32 * sub;
                len = len < 0 ? 0 : len > 32 ? 32 : len;
            }
        }
        int4 na = make_int4(0, 0, 0, 0), nb = na, nc = na;
        auto fetch = [&](int j) {
            const int64_t packet = __shfl_sync(0xffffffffu, at, j);
            const int m = __shfl_sync(0xffffffffu, len, j);
            if (lane < m) {
                const int4* __restrict__ p = packets + (packet + lane) * (kPacketWords / 4);
                na = __ldg(p); nb = __ldg(p + 1); nc = __ldg(p + 2);
            }
        };
        fetch(0);
        for (int j = 0; j < per_warp; ++j) {
            const int n = __shfl_sync(0xffffffffu, len, j);
            const int4 pa = na, pb = nb, pc = nc;
            if (j + 1 < per_warp) fetch(j + 1);     // one batch ahead
            if (n == 0) continue;
            uint32_t slot = 0;
            int off = 0, hoff = 0;
            float f[3] = {0.f, 0.f, 0.f}, fh[3] = {0.f, 0.f, 0.f}, gs = 0.f, hs = 0.f;
            float basis[BD > 0 ? BD : 1] = {};
            const bool want_grad = !HESS || to.grad != nullptr;
            if (lane < n) {
                slot = (uint32_t)pa.x;
                const int64_t ray = pa.y;
                const float q[3] = {__int_as_float(pa.z), __int_as_float(pa.w),
                                    __int_as_float(pb.x)};
                const float h[3] = {__int_as_float(pb.y), __int_as_float(pb.z),
                                    __int_as_float(pb.w)};
                const float dd = __int_as_float(pc.x);
                float one_minus_s = 0.f;
                // Gauss-Newton diagonal with a softplus density: the reference adds, per
                // channel, (d out / d raw)^2 + (d out / d density) * softplus'' with its own
                // formula for the second term (svox/csrc/rt_kernel.cu:683-693); dd already
                // holds softplus' = s
                if (HESS && opt.density_softplus)
                    one_minus_s =
                        1.f - sigmoid_ref(__ldg(tr.data + (int64_t)slot * K + (K - 1)) - 1);
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) {
                    const float rest = h[ch] - __ldg(to.fwd_out + 3 * ray + ch);
                    if (want_grad) {
                        const float g = __ldg(to.grad_out + 3 * ray + ch);
                        f[ch] = q[ch] * g * d_rgb_pad;
                        gs += rest * g;
                    }
                    if (HESS) {
                        fh[ch] = q[ch] * d_rgb_pad;
                        const float ds = dd * rest;
                        hs += ds * ds + ds * one_minus_s;
                    }
                }
                gs *= dd;
                // the record is placed in the row as in memory (offset within the first
                // 16-byte word), zeros around it
                off = record_offset<K>(to.grad, slot);
                hoff = HESS ? record_offset<K>(to.hess, slot) : 0;
                if constexpr (BD > 0) {
                    const float vdir[3] = {__int_as_float(pc.y), __int_as_float(pc.z),
                                           __int_as_float(pc.w)};
                    colour_basis<BD, LOBES>(tr, opt, vdir, basis);
#pragma unroll
                    for (int k = 0; k < BD; ++k)
                        if (k < opt.min_comp || k > opt.max_comp) basis[k] = 0.f;
                }
            }
            float* row = sm.rows + lane * Shape::STRIDE;
            auto expand = [&](float* __restrict__ r, int o, bool square) {
                float v[K];
#pragma unroll
                for (int ch = 0; ch < 3; ++ch) {
                    if constexpr (BD == 0) {
                        v[ch] = square ? fh[ch] * fh[ch] : f[ch];
                    } else {
#pragma unroll
                        for (int k = 0; k < BD; ++k) {
                            const float w = basis[k] * (square ? fh[ch] : f[ch]);
                            v[ch * BD + k] = square ? w * w : w;
                        }
                    }
                }
                v[K - 1] = square ? hs : gs;
                if (Shape::ALIGNED) {
#pragma unroll
                    for (int w = 0; w < K / 4; ++w)
                        reinterpret_cast<float4*>(r)[w] =
                            make_float4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        if (i < o) r[i] = 0.f;
                        if (o + K + i < 4 * Shape::WORDS) r[o + K + i] = 0.f;
                    }
#pragma unroll
                    for (int w = 0; w < K; ++w) r[o + w] = v[w];
                }
            };
            if (lane < n && want_grad) expand(row, off, false);
            __syncwarp();
            // groups of lanes add consecutive 16-byte words of a record
            auto flush = [&](float* __restrict__ out, const float* rows, int offset) {
                const bool vec_ok = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
                const int sub = lane / Shape::GROUP, w = lane % Shape::GROUP;
#pragma unroll
                for (int p = 0; p < Shape::GROUP; ++p) {
                    const int k = p * Shape::RPP + sub;
                    const uint32_t sl = __shfl_sync(0xffffffffu, slot, k);
                    const int o = __shfl_sync(0xffffffffu, offset, k);
                    if (k < n && w < Shape::WORDS)
                        flush_word<K>(out + (size_t)sl * K, o, w,
                                      reinterpret_cast<const float4*>(rows + k * Shape::STRIDE)[w],
                                      vec_ok, pol_keep);
                }
            };
            if (want_grad) flush(to.grad, sm.rows, off);
            __syncwarp();
            if constexpr (HESS) {       // through the same rows
                if (lane < n) expand(row, hoff, true);
                __syncwarp();
                flush(to.hess, sm.rows, hoff);
                __syncwarp();
            }
        }
    };
    // Clearing is spread between the units of adding where these are large, and for records of up to 28
    // floats.  Scatter alone (512^3 shell, us, before / between): 2^20 rays RGBA 935 / 938, SH4 1729 / 1719,
    // SH9 1931 / 1891; views of 1000x1000 and 1600x1600 pixels, SH9, 915 / 887 and 1668 / 1635; but 2^19
    // rays SH16 2156 / 2182, a view of 1200x1200 2183 / 2216.  Small units then hold up the next bin:
    // 2^18 rays SH9 746 / 792, `se_grad` of 100 000 rays 1.12 / 1.28 ms.
    ordered_units<BLOCK>(s_units, counters, lo_bin, hi_bin, groups_before,
                         WARPS * per_warp / per_group, ((int64_t)1 << log[2]) * K,
                         sorted ? to.zero_slots * K : 0, K <= 28 && per_warp >= 4, count, clear, work);
}

}  // namespace svoxb
