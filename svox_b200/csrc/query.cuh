// Point query kernels: query_vertical and its backward.
//
// Replaces query_single_kernel / query_single_kernel_backward of the
// reference (svox/csrc/svox_kernel.cu:56-78).  The reference copies each
// point's K-float record with a per-thread scalar loop, so every warp
// instruction touches 32 different cache lines on both sides.  Here a thread
// still descends for its own point, but the records of a warp's 32 points
// are then moved by the whole warp, so that loads and stores run along rows.
// The backward works on the leaf ids that the forward found.
//
// HBM roofline per point: 12 B in + K*4 B gathered + K*4 B written + 8 B id
// (+ one 4-B child entry per level below the jump table, L2 resident).  2^24 points over 256^3
// leaves of 49 floats, 268 of the 196 bytes per record read (64-byte pieces): 1.75 -> 1.63 ms.
// Backward: 3.43 ms (clear, then reductions at random) -> 2.57 (binned) -> 2.0 (summed by tiles, see
// below).
#pragma once

#include "common.cuh"
#include "binned.cuh"
#include "tiles.cuh"

namespace svoxb {

constexpr int kQueryBlock = 256;

struct TreeArgs {
    const float* __restrict__ data;
    const int32_t* __restrict__ child;
    const float* __restrict__ offset;
    const float* __restrict__ scaling;
    int64_t M;
    int32_t N;
    int32_t K;
    float* weight_accum;      // forward render only (null: off)
    int32_t weight_accum_max;
    int32_t extra_cols;       // row length of `extra`
    const float* __restrict__ extra;   // lobe parameters of the SG / ASG colour bases
};

static inline TreeArgs tree_args(const svoxb_tree* t) {
    return TreeArgs{t->data, t->child, t->offset, t->scaling, t->M, t->N, t->K,
                    t->weight_accum, t->weight_accum_max, t->extra_cols, t->extra_data};
}

// One sample's weight into the accumulator of its leaf (svox/csrc/rt_kernel.cu:298-304).
// Weights are >= 0 unless the density is negative; for those the maximum goes through a
// compare-and-swap like the reference's (svox/csrc/include/common.cuh:152-161).
__device__ __forceinline__ void accumulate_weight(const TreeArgs& tr, int64_t slot, float w) {
    float* p = tr.weight_accum + slot;
    if (!tr.weight_accum_max) {
        atomicAdd(p, w);
    } else if (w >= 0.f) {
        // non-negative floats order like their bit patterns; the buffer starts at +0
        if (__float_as_int(*reinterpret_cast<volatile float*>(p)) < __float_as_int(w))
            atomicMax(reinterpret_cast<int*>(p), __float_as_int(w));
    } else {
        unsigned* u = reinterpret_cast<unsigned*>(p);
        unsigned old = *u, assumed;
        int guard = 0;
        do {
            assumed = old;
            old = atomicCAS(u, assumed, __float_as_uint(fmaxf(w, __uint_as_float(assumed))));
        } while (old != assumed && ++guard < 1024);
    }
}

__device__ __forceinline__ int64_t locate_point(const TreeArgs& tr, const TopTable& top,
                                                const float* __restrict__ pts, int64_t i) {
    const float px = to_tree(__ldg(pts + 3 * i + 0), __ldg(tr.offset + 0), __ldg(tr.scaling + 0));
    const float py = to_tree(__ldg(pts + 3 * i + 1), __ldg(tr.offset + 1), __ldg(tr.scaling + 1));
    const float pz = to_tree(__ldg(pts + 3 * i + 2), __ldg(tr.offset + 2), __ldg(tr.scaling + 2));
    LeafHit hit;
    const bool ok = (tr.N == 2) ? descend2(tr.child, tr.M, top, px, py, pz, hit)
                                : descendN(tr.child, tr.M, tr.N, px, py, pz, hit);
    return ok ? hit.slot : -1;
}

// Records are fetched in 64-byte pieces of L2 lines (without the hint the L2 reads 128 bytes for
// each of these scattered pieces).
__device__ __forceinline__ float ld_row(const float* a) {
    float v;
    asm volatile("ld.global.nc.L2::64B.f32 %0, [%1];" : "=f"(v) : "l"(a));
    return v;
}

// Forward: the records of the points' leaves, row by row.  G lanes copy a row, STEPS elements
// each (0: as many as it takes); PASSES of them are under way at a time, loads first.  A flat walk
// over the warp's output block, with a division's worth of index arithmetic per element, spent
// 74 instructions per point of 49 floats and 73 % of the issue slots.
template <int G, int STEPS>
__global__ void __launch_bounds__(kQueryBlock)
query_kernel(TreeArgs tr, TopTable top, const float* __restrict__ pts, int64_t Q,
             float* __restrict__ values_out, int64_t* __restrict__ ids_out) {
    const int64_t i = (int64_t)blockIdx.x * kQueryBlock + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int64_t slot = -1;
    if (i < Q) {
        slot = locate_point(tr, top, pts, i);
        if (ids_out != nullptr) ids_out[i] = slot;      // -1: not a tree
    }
    const int64_t wb = i - lane;            // first point of this warp
    if (values_out == nullptr || wb >= Q) return;
    const int K = tr.K;
    const int sub = lane / G, e = lane % G;
    constexpr int ROWS = 32 / G;            // rows per pass
    constexpr int N = STEPS > 0 ? STEPS : 1;
    constexpr int PASSES = G < 8 / N ? G : 8 / N;
    const int n = (int)(Q - wb < 32 ? Q - wb : 32);
    float* __restrict__ out = values_out + wb * K;
    for (int base = 0; STEPS > 0 ? base == 0 : base < K; base += G) {
#pragma unroll 1
        for (int p0 = 0; p0 < G; p0 += PASSES) {
            float v[PASSES][N];
#pragma unroll
            for (int p = 0; p < PASSES; ++p) {
                const int k = (p0 + p) * ROWS + sub;
                const int64_t s = __shfl_sync(0xffffffffu, slot, k);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    v[p][j] = 0.f;
                    if (s >= 0 && base + e + j * G < K)
                        v[p][j] = ld_row(tr.data + s * K + (base + e + j * G));
                }
            }
#pragma unroll
            for (int p = 0; p < PASSES; ++p) {
                const int k = (p0 + p) * ROWS + sub;
                // (a point without a leaf -- not a tree -- leaves its row as it is)
                const bool there = __shfl_sync(0xffffffffu, slot, k) >= 0;
#pragma unroll
                for (int j = 0; j < N; ++j)
                    if (k < n && there && base + e + j * G < K)
                        out[k * K + (base + e + j * G)] = v[p][j];
            }
        }
    }
}

// The same for records of up to kStagedRow floats, through shared memory: `per` rows of a warp at a
// time are requested with cp.async, as 16-byte words where records are aligned (VEC), else as
// floats, and leave as one stretch in 16-byte words.  `per` rows of a warp are under way at once, 32 up
// to 28 floats and 4 of more than 112, and as 16-byte words a quarter of the requests are made.
// Measured (2^22 points, us; row by row / staged):
//   words    8 floats 99 / 103, 12: 130 / 127, 16: 142 / 132, 20: 266 / 174, 28: 304 / 251, 76: 483 / 478,
//            100: 1050 / 606, 128: 685 / 606; 4 (RGBA) 76 / 78
//   floats   13 floats 136 / 144, 49: 344 / 395, 97: 1202 / 730, 129: 1477 / 840, 144: 939 / 888, 160: 893
//            / 950, 192: 1101 / 1099, 200: 1512 / 1255, 208: 1424 / 1280, 223: 2752 / 1378, 224: 1304 / 1338
// So records up to 8 floats, unaligned ones up to 96, and long ones of a multiple of 32 floats, which
// fill every request of a warp, go row by row.
constexpr int kStagedRow = 224;
constexpr int kStagedFloats = 896;       // per warp
template <int G, int STEPS, bool VEC>
__global__ void __launch_bounds__(kQueryBlock)
query_staged_kernel(TreeArgs tr, TopTable top, const float* __restrict__ pts, int64_t Q,
                    float* __restrict__ values_out, int64_t* __restrict__ ids_out, int per) {
    extern __shared__ __align__(16) float s_rows[];
    const int64_t i = (int64_t)blockIdx.x * kQueryBlock + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int64_t slot = -1;
    if (i < Q) {
        slot = locate_point(tr, top, pts, i);
        if (ids_out != nullptr) ids_out[i] = slot;      // -1: not a tree
    }
    const int64_t wb = i - lane;            // first point of this warp
    if (values_out == nullptr || wb >= Q) return;
    constexpr int W = VEC ? 4 : 1;
    const int K = tr.K, words = K / W;
    const int sub = lane / G, e = lane % G;
    constexpr int ROWS = 32 / G;
    const int n = (int)(Q - wb < 32 ? Q - wb : 32);
    float* const mine = s_rows + (threadIdx.x >> 5) * per * K;
    float* __restrict__ out = values_out + wb * K;
    // (a point without a leaf -- not a tree -- leaves its row as it is)
    const bool whole = __all_sync(0xffffffffu, i >= Q || slot >= 0) &&
                       (reinterpret_cast<uintptr_t>(values_out) & 15) == 0;
    for (int first = 0; first < n; first += per) {
        const int until = n - first < per ? n - first : per;
#pragma unroll 4
        for (int p = 0; p < until; p += ROWS) {
            const int k = p + sub;
            const int64_t s = __shfl_sync(0xffffffffu, slot, first + k);
            const float* const src = tr.data + s * K + e * W;
            float* const to = mine + k * K + e * W;
            if (k < until && s >= 0) {
#pragma unroll
                for (int j = 0; j < STEPS; ++j) {
                    if (e + j * G >= words) continue;
                    const unsigned a = (unsigned)__cvta_generic_to_shared(to + j * G * W);
                    if (VEC)
                        asm volatile("cp.async.cg.shared.global.L2::64B [%0], [%1], 16;" ::"r"(a),
                                     "l"(src + j * G * W) : "memory");
                    else
                        asm volatile("cp.async.ca.shared.global.L2::64B [%0], [%1], 4;" ::"r"(a),
                                     "l"(src + j * G * W) : "memory");
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        const int floats = until * K;
        if (whole) {
            for (int f = lane; f < floats / 4; f += 32)
                reinterpret_cast<float4*>(out)[f] = reinterpret_cast<const float4*>(mine)[f];
            if (lane < (floats & 3)) out[(floats & ~3) + lane] = mine[(floats & ~3) + lane];
        } else {
            for (int k = 0; k < until; ++k) {
                const int64_t s = __shfl_sync(0xffffffffu, slot, first + k);
                for (int c = lane; s >= 0 && c < K; c += 32) out[k * K + c] = mine[k * K + c];
            }
        }
        out += floats;
        __syncwarp();
    }
}

// Overwrites the first Kv floats of each point's record with its row of `values`
// (assign_single_kernel, svox/csrc/svox_kernel.cu:80-89; points that share a leaf race, as in the
// reference).
__global__ void __launch_bounds__(kQueryBlock)
assign_kernel(TreeArgs tr, TopTable top, const float* __restrict__ pts, int64_t Q,
              const float* __restrict__ values, float* __restrict__ data_out, int Kv) {
    const int64_t i = (int64_t)blockIdx.x * kQueryBlock + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int64_t slot = i < Q ? locate_point(tr, top, pts, i) : -1;
    const int64_t wb = i - lane;
    if (wb >= Q) return;
    // lanes walk the warp's block of rows in order: coalesced reads, and writes that are
    // contiguous within each record
    const int nvalid = (int)((Q - wb) < 32 ? (Q - wb) : 32);
    const int total = nvalid * Kv;
    int p = 0, e = lane;
    while (e >= Kv) { e -= Kv; ++p; }
    for (int base = 0; base < total; base += 32) {        // warp-uniform trip count
        const int j = base + lane;
        const int64_t s = __shfl_sync(0xffffffffu, slot, p < nvalid ? p : nvalid - 1);
        if (j < total && s >= 0) data_out[s * tr.K + e] = __ldg(values + wb * Kv + j);
        e += 32;
        while (e >= Kv) { e -= Kv; ++p; }
    }
}

// calc_corner_kernel (svox/csrc/svox_kernel.cu:91-115): the lower corner of cell (node, i, j, k)
// in tree-local coordinates, by walking parent_depth up to the root with the reference's
// add-then-divide per level (for N = 3 the roundings of that order are part of the result).
// parent_depth is (M, 2): packed index of the parent cell, depth.
__global__ void calc_corners_kernel(const int32_t* __restrict__ parent_depth, int64_t M, int N,
                                    const int64_t* __restrict__ indexer, int64_t Q,
                                    float* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Q) return;
    int64_t node = indexer[4 * i];
    int c[3] = {(int)indexer[4 * i + 1], (int)indexer[4 * i + 2], (int)indexer[4 * i + 3]};
    float r[3] = {0.f, 0.f, 0.f};
    const float fn = (float)N;
    for (int level = 0;; ++level) {
        if (node < 0 || node >= M || level > 64) {   // not a tree: reported, never followed
            report(SVOXB_ERR_TREE);
            break;
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) r[a] = __fdiv_rn(__fadd_rn(r[a], (float)c[a]), fn);
        if (node == 0) break;
        int32_t packed = __ldg(parent_depth + 2 * node);
        for (int a = 2; a >= 0; --a) {
            c[a] = packed % N;
            packed /= N;
        }
        node = packed;
    }
    out[3 * i + 0] = r[0];
    out[3 * i + 1] = r[1];
    out[3 * i + 2] = r[2];
}

// Query, or with `rows` assignment.
static int launch_query(const svoxb_tree* tree, const float* indices, int64_t Q,
                        float* values_out, int64_t* ids_out, const float* rows, float* data_out,
                        int Kv, cudaStream_t stream) {
    if (Q == 0) return SVOXB_OK;
    if (!indices) return SVOXB_ERR_NULL;
    if ((Q + kQueryBlock - 1) / kQueryBlock > 0x7fffffffLL) return SVOXB_ERR_TOO_LARGE;
    // The jump table saves a point its upper levels, at a cost of one walk per cell: it has at
    // most a quarter as many cells as there are points, and few points go without.
    TopScratch top;
    int level = 0;
    while (level < 7 && Q >= (int64_t)4 << (3 * (level + 1))) ++level;
    int st = level >= 5 ? top.build(tree, level, stream) : (int)SVOXB_OK;
    if (st) return st;
    const TopTable tt{top.cells, top.level};
    const unsigned grid = (unsigned)((Q + kQueryBlock - 1) / kQueryBlock);
    auto forward = [&](auto kernel) {
        kernel<<<grid, kQueryBlock, 0, stream>>>(tree_args(tree), tt, indices, Q, values_out,
                                                 ids_out);
    };
    const int K = tree->K;
    const bool vec = K % 4 == 0 && reinterpret_cast<uintptr_t>(tree->data) % 16 == 0;
    int per = 32;
    while (per * K > kStagedFloats && per > 4) per /= 2;
    auto staged = [&](auto kernel) {
        kernel<<<grid, kQueryBlock, kQueryBlock / 32 * per * K * sizeof(float), stream>>>(
            tree_args(tree), tt, indices, Q, values_out, ids_out, per);
    };
    if (rows != nullptr)
        assign_kernel<<<grid, kQueryBlock, 0, stream>>>(tree_args(tree), tt, indices, Q, rows,
                                                        data_out, Kv);
    else if (values_out == nullptr || K > kStagedRow || (K > 128 && K % 32 == 0))
        forward(query_kernel<32, 0>);
    else if (vec && K > 8 && K <= 16) staged(query_staged_kernel<4, 1, true>);
    else if (vec && K > 16 && K <= 32) staged(query_staged_kernel<8, 1, true>);
    else if (vec && K > 32 && K <= 128) staged(query_staged_kernel<32, 1, true>);
    else if (K <= 2) forward(query_kernel<2, 1>);
    else if (K <= 4) forward(query_kernel<4, 1>);
    else if (K <= 8) forward(query_kernel<8, 1>);
    else if (K <= 16) forward(query_kernel<16, 1>);
    else if (K <= 32) forward(query_kernel<32, 1>);
    else if (K <= 64) forward(query_kernel<32, 2>);
    else if (K <= 96) forward(query_kernel<32, 3>);
    else staged(query_staged_kernel<32, 7, false>);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

// ---------------------------------------------------------------------------
// Backward of the query: row q of the upstream gradient is added into record ids[q].

// 32 rows of a warp.  Groups of G lanes take a row each; lane w adds the 16-byte word w of the
// record's place in memory (with zeros where the word reaches beyond the record), a quarter of
// the requests of scalar atomics.  `slot` < 0: no row.
template <int G>
__device__ __forceinline__ void add_rows(int64_t slot, int64_t row, int n,
                                         const float* __restrict__ rows, int K,
                                         float* __restrict__ grad, int64_t n_floats, bool vec_ok,
                                         uint64_t pol) {
    const int lane = threadIdx.x & 31;
    const int sub = lane / G, w = lane % G;
#pragma unroll 4
    for (int p = 0; p < G; ++p) {
        const int k = p * (32 / G) + sub;
        const int64_t s = __shfl_sync(0xffffffffu, slot, k);
        const int64_t r = __shfl_sync(0xffffffffu, row, k);
        if (k >= n || s < 0) continue;
        const float* __restrict__ src = rows + r * K;
        const int64_t first = s * K;
        const int off = vec_ok ? (int)(first & 3) : 0;
        for (int word = w; 4 * word < off + K; word += G) {
            const int e = 4 * word - off;
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = e + i >= 0 && e + i < K ? ld_row(src + e + i) : 0.f;
            float* to = grad + first + e;
            if (vec_ok && first + e + 4 <= n_floats) {
                red_add_v4_hint(to, v[0], v[1], v[2], v[3], pol);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (e + i >= 0 && e + i < K) atomicAdd(to + i, v[i]);
            }
        }
    }
}

template <int G>
__global__ void __launch_bounds__(kQueryBlock)
scatter_rows_kernel(const int64_t* __restrict__ ids, int64_t Q, const float* __restrict__ rows,
                    int K, float* __restrict__ grad, int64_t n_slots) {
    const int64_t i = (int64_t)blockIdx.x * kQueryBlock + threadIdx.x;
    const int64_t wb = i - (threadIdx.x & 31);
    if (wb >= Q) return;
    int64_t slot = i < Q ? ids[i] : -1;
    if (slot >= n_slots) slot = -1;
    add_rows<G>(slot, i, 32, rows, K, grad, n_slots * K,
                (reinterpret_cast<uintptr_t>(grad) & 15) == 0, l2_policy_stream());
}

// Many rows into a gradient that outgrows the L2: the points are sorted into bins first (count,
// place), then their rows are added bin by bin, each bin cleared on the way (binned.cuh).
struct RowBins {
    int32_t* count;      // [kMaxBins]
    int32_t* cursor;     // [kMaxBins]
    UnitCounters units;
    int2* pair;          // [Q] {slot, row}
    int shift, n_bins;
};
constexpr int kBinRows = 2048;       // points a block sorts at a time

__global__ void __launch_bounds__(256)
count_rows_kernel(const int64_t* __restrict__ ids, int64_t Q, int64_t n_slots, RowBins b) {
    __shared__ int s_count[kMaxBins];
    for (int i = threadIdx.x; i < kMaxBins; i += 256) s_count[i] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < Q; i += (int64_t)gridDim.x * 256) {
        const int64_t slot = ids[i];
        if (slot >= 0 && slot < n_slots) atomicAdd(&s_count[(int)(slot >> b.shift)], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < b.n_bins; i += 256)
        if (s_count[i]) atomicAdd(b.count + i, s_count[i]);
}

__global__ void __launch_bounds__(256)
place_rows_kernel(const int64_t* __restrict__ ids, int64_t Q, int64_t n_slots, RowBins b) {
    __shared__ int s_first[kMaxBins], s_count[kMaxBins];
    for (int i = threadIdx.x; i < kMaxBins; i += 256) s_first[i] = b.count[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int i = 0; i < kMaxBins; ++i) {
            const int n = s_first[i];
            s_first[i] = run;
            run += n;
        }
    }
    for (int64_t tile = blockIdx.x; tile * kBinRows < Q; tile += gridDim.x) {
        __syncthreads();
        for (int i = threadIdx.x; i < kMaxBins; i += 256) s_count[i] = 0;
        __syncthreads();
        int slot[kBinRows / 256], rank[kBinRows / 256];
#pragma unroll
        for (int j = 0; j < kBinRows / 256; ++j) {
            const int64_t i = tile * kBinRows + 256 * j + threadIdx.x;
            const int64_t s = i < Q ? ids[i] : -1;
            slot[j] = s >= 0 && s < n_slots ? (int)s : -1;
            rank[j] = slot[j] >= 0 ? atomicAdd(&s_count[slot[j] >> b.shift], 1) : 0;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < b.n_bins; i += 256)
            if (s_count[i] > 0) s_count[i] = s_first[i] + atomicAdd(b.cursor + i, s_count[i]);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kBinRows / 256; ++j)
            if (slot[j] >= 0)
                b.pair[s_count[slot[j] >> b.shift] + rank[j]] =
                    make_int2(slot[j], (int)(tile * kBinRows + 256 * j + threadIdx.x));
    }
}

template <int G>
__global__ void __launch_bounds__(kQueryBlock)
scatter_binned_rows_kernel(int64_t Q, const float* __restrict__ rows, int K,
                           float* __restrict__ grad, int64_t n_slots, RowBins b, int per_warp) {
    __shared__ UnitShared s_units;
    const int lane = threadIdx.x & 31;
    const uint64_t pol_keep = l2_policy_keep();
    auto clear = [&](int64_t from, int64_t until) {
        const int4 none = make_int4(0, 0, 0, 0);
        int64_t i = from + 4 * threadIdx.x;
        for (; i + 4 <= until; i += 4 * kQueryBlock) st_hint16(grad + i, none, pol_keep);
        for (; i < until; ++i) grad[i] = 0.f;      // the end of a buffer of odd length
    };
    auto work = [&](int first, int end) {
        first += (threadIdx.x >> 5) * per_warp * 32;
        for (int j = 0; j < per_warp; ++j, first += 32) {
            const int n = end - first < 32 ? end - first : 32;
            if (n <= 0) break;
            int2 p = make_int2(0, 0);
            if (lane < n) p = __ldg(b.pair + first + lane);
            add_rows<G>(p.x, p.y, n, rows, K, grad, n_slots * K, true, pol_keep);
        }
    };
    ordered_units<kQueryBlock>(s_units, b.units, 0, b.n_bins, 0, kQueryBlock * per_warp,
                               ((int64_t)1 << b.shift) * K, n_slots * K, false,
                               [&](int i) { return b.count[i]; }, clear, work);
}

// Long rows into a gradient far larger than the L2: the points are sorted by tile of the gradient, and
// a block adds up the rows of a tile's points (tiles.cuh).
constexpr int kPlaceBlock = 512;
constexpr int kPlaceEach = 16;       // points a thread places at a time

// Items per range of rows of the points.
__global__ void __launch_bounds__(kPlaceBlock)
count_ranges_kernel(const int64_t* __restrict__ ids, TileLists t) {
    extern __shared__ int s_count[];
    for (int i = threadIdx.x; i < t.n_ranges; i += kPlaceBlock) s_count[i] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * kPlaceBlock + threadIdx.x; i < t.n_items;
         i += (int64_t)gridDim.x * kPlaceBlock) {
        const int64_t slot = ids[i];
        if (slot >= 0 && slot < t.n_rows) atomicAdd(s_count + (int)(slot >> t.shift), 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < t.n_ranges; i += kPlaceBlock)
        if (s_count[i]) atomicAdd(t.in_range + i, s_count[i]);
    if (last_block(t.head + 4)) cut_ranges<kPlaceBlock>(t);
}

// Items per tile of the points, where these are not the ranges.
__global__ void __launch_bounds__(kPlaceBlock)
count_tiles_kernel(const int64_t* __restrict__ ids, TileLists t) {
    extern __shared__ int s_count[];
    const int n_tiles = t.head[3];
    if (n_tiles == t.n_ranges) return;
    for (int i = threadIdx.x; i < n_tiles; i += kPlaceBlock) s_count[i] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * kPlaceBlock + threadIdx.x; i < t.n_items;
         i += (int64_t)gridDim.x * kPlaceBlock) {
        const int64_t slot = ids[i];
        if (slot >= 0 && slot < t.n_rows) atomicAdd(s_count + t.tile_of(slot), 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_tiles; i += kPlaceBlock)
        if (s_count[i]) atomicAdd(t.count + i, s_count[i]);
    if (last_block(t.head + 5)) list_tiles<kPlaceBlock>(t, t.count);
}

// Lists the points {slot, row} tile by tile.  0.19 ms for 2^24 points and 4681 tiles, the same with
// 256 to 1024 threads.
__global__ void __launch_bounds__(kPlaceBlock)
place_tiles_kernel(const int64_t* __restrict__ ids, TileLists t, int2* __restrict__ pair, int K,
                   float* __restrict__ grad) {
    extern __shared__ int s_count[];
    clear_hot_tiles(t, K, grad);
    const int n_tiles = t.head[3];
    constexpr int64_t each = kPlaceEach * kPlaceBlock;
    for (int64_t first = blockIdx.x * each; first < t.n_items; first += gridDim.x * each) {
        __syncthreads();
        for (int i = threadIdx.x; i < n_tiles; i += kPlaceBlock) s_count[i] = 0;
        __syncthreads();
        int slot[kPlaceEach], rank[kPlaceEach];
#pragma unroll
        for (int j = 0; j < kPlaceEach; ++j) {
            const int64_t i = first + kPlaceBlock * j + threadIdx.x;
            const int64_t s = i < t.n_items ? ids[i] : -1;
            slot[j] = s >= 0 && s < t.n_rows ? (int)s : -1;
        }
#pragma unroll
        for (int j = 0; j < kPlaceEach; ++j)
            rank[j] = slot[j] >= 0 ? atomicAdd(s_count + t.tile_of(slot[j]), 1) : 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n_tiles; i += kPlaceBlock)
            if (s_count[i] > 0) s_count[i] = atomicAdd(t.end + i, s_count[i]);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPlaceEach; ++j)
            if (slot[j] >= 0)
                pair[rank[j] + s_count[t.tile_of(slot[j])]] =
                    make_int2(slot[j], (int)(first + kPlaceBlock * j + threadIdx.x));
    }
}

// A 16-byte word into shared memory, asynchronously, in 64-byte pieces of L2 lines.
__device__ __forceinline__ void copy_word(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global.L2::64B [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}

// Items of a tile from which its rows, and the zeros between them, leave through StreamWriter:
// fewer items leave most of the tile to few of the warps.
constexpr int kStreamItems = 32;
constexpr int kStageWords = 104;     // 16-byte words of rows a warp has under way per stage

// `grad` is 16-byte aligned.  Warps take equal shares of a tile's sorted items; lane e of a warp holds columns e, e + 32, ... of
// the row being summed (N of them; further columns in further passes).  Rows come in as the 16-byte
// words that cover them, a stage of some rows ahead of the one being summed; finished rows, and
// zeros between them, leave through a StreamWriter.  2^24 rows of 49 floats into 3.76 GB: 2.41 ms
// with the gradient cleared and added to bin by bin, 1.78 so.  Bound: issue slots (79 % used, 69
// instructions per row in a capture of 2^22 rows); without the stores it takes 0.95 ms, and 2.05 with a row's floats stored
// one by one; unrolled by the row it outgrew the instruction cache (4.6 ms).
template <int N>
__global__ void __launch_bounds__(kOwnBlock, 2)
own_rows_kernel(const float* __restrict__ rows, uint32_t last_id, int K,
                float* __restrict__ grad, TileLists t, const int2* __restrict__ pair) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ float s_carry[kOwnWarps * 32 * N];
    __shared__ int s_state[kOwnWarps];
    const TileSort sorted(s_raw);
    // (through a shuffle, so that the compiler knows it to be the same in a warp: loops over a warp's
    // items then need no code for divergence)
    const int me = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), e = threadIdx.x & 31;
    float* const stages = reinterpret_cast<float*>(s_raw + TileSort::kBytes);
    float* const stage = stages + me * (2 * 4 * kStageWords);
    StreamWriter writer;
    writer.buf = stages + kOwnWarps * (2 * 4 * kStageWords) + me * (2 * StreamWriter::kPiece);
    writer.clear();
    const uint32_t pitch = 4u * (uint32_t)K;
    const bool one_pass = K <= 32 * N;
    owned_units(t, [&](int tile, int first, int last, bool hot) {
        const int64_t row0 = t.first_row(tile);
        const int shift = t.tile_shift(tile);
        if (row0 >= t.n_rows) return;            // the last range may reach beyond the buffer
        const int n_rows = (int)(t.n_rows - row0 < (1 << shift) ? t.n_rows - row0
                                                                : (int64_t)1 << shift);
        float* __restrict__ out = grad + row0 * K;
        bool store = !hot;          // rows are written, else added to
        do {
            const int n = last - first < kOwnItems ? last - first : kOwnItems;
            sorted.sort(n, shift, [&](int i) {
                const int2 p = __ldg(pair + first + i);
                return make_int2(p.x - (int)row0, p.y);
            });
            const bool stream = store && one_pass && n >= kStreamItems;
            if (store && !stream) sorted.clear_empty(n_rows, K, out);
            const int lo = n * me / kOwnWarps, hi = n * (me + 1) / kOwnWarps;
            for (int base = 0; base < K; base += 32 * N) {
                const int cols = K - base < 32 * N ? K - base : 32 * N;
                const uintptr_t src = reinterpret_cast<uintptr_t>(rows + base);
                // words per row; whether a row may not need its last one; rows per stage; the
                // lane's words of a stage
                const bool same = K % 4 == 0;
                const int words = same ? ((int)(src >> 2 & 3) + cols + 3) / 4 : (cols + 6) / 4;
                const bool loose = !same && cols % 4 != 1;
                const int per = kStageWords / words < 32 ? kStageWords / words : 32;
                constexpr int COPIES = (kStageWords + 31) / 32;
                int at_item[COPIES], at_word[COPIES];
#pragma unroll
                for (int p = 0; p < COPIES; ++p) {
                    const int w = 32 * p + e;
                    at_item[p] = w < per * words ? w / words : 1 << 16;
                    at_word[p] = 16 * (w % words);
                }
                float acc[N];
#pragma unroll
                for (int j = 0; j < N; ++j) acc[j] = 0.f;
                auto issue = [&](int i, float* to) {
#pragma unroll
                    for (int p = 0; p < COPIES; ++p) {
                        const int k = i + at_item[p];
                        if (k < hi) {
                            const uint32_t id = sorted.item[k];
                            const uintptr_t a =
                                ((src + (uint64_t)id * pitch) & ~(uintptr_t)15) + at_word[p];
                            if (loose && id == last_id && a >= src + (uint64_t)id * pitch + 4 * cols)
                                continue;                        // beyond the buffer
                            copy_word(to + 4 * (32 * p + e), reinterpret_cast<const void*>(a));
                        }
                    }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                };
                auto hand_on = [&](int state) {
                    if (e == 0) s_state[me] = state;
#pragma unroll
                    for (int j = 0; j < N; ++j) s_carry[me * (32 * N) + e + j * 32] = acc[j];
                };
                auto flush = [&](int r) {
                    if (stream) {
                        writer.skip_to(r * K);
                        writer.append<N>(acc, K);
                    } else {
                        float* const to = out + (r * K + base + e);
#pragma unroll
                        for (int j = 0; j < N; ++j) {
                            if (e + 32 * j < cols) {
                                if (store) to[32 * j] = acc[j];
                                else atomicAdd(to + 32 * j, acc[j]);
                            }
                        }
                    }
                };
                if (e == 0) s_state[me] = lo < hi ? kCarryNone : kCarrySkip;
                // the first run began with an earlier warp
                const int before = lo > 0 ? sorted.row[lo - 1] : -1;
                writer.begin(out, (before + 1) * K);
                bool head = lo > 0 && lo < hi && before == sorted.row[lo];
                issue(lo, stage);
                int buf = 0;
                for (int i = lo; i < hi; i += per, buf ^= 1) {
                    issue(i + per, stage + (buf ^ 1) * (4 * kStageWords));
                    const int k = i + e, m = hi - i < per ? hi - i : per;
                    bool ends = false;
                    int at_row = 0;
                    if (e < m) {
                        ends = k + 1 == n || sorted.row[k + 1] != sorted.row[k];
                        at_row = e * words * 4 +
                                 ((int)((src + (uint64_t)sorted.item[k] * pitch) >> 2) & 3);
                    }
                    unsigned mask = __ballot_sync(0xffffffffu, ends);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                    __syncwarp();
                    const float* const in = stage + buf * (4 * kStageWords) + e;
                    for (int a = 0;;) {
                        const int stop = mask != 0u ? __ffs(mask) : m;
#pragma unroll 1
                        for (; a < stop; ++a) {
                            // (lanes beyond the row's columns add what lies there and drop it)
                            const float* const row = in + __shfl_sync(0xffffffffu, at_row, a);
#pragma unroll
                            for (int j = 0; j < N; ++j) acc[j] += row[32 * j];
                        }
                        if (mask == 0u) break;
                        mask &= mask - 1u;                               // a run ends here
                        if (head) hand_on(kCarryEnds);
                        else flush(sorted.row[i + a - 1]);
                        head = false;
#pragma unroll
                        for (int j = 0; j < N; ++j) acc[j] = 0.f;
                    }
                    __syncwarp();
                }
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                // the last run goes on with the next warp
                const bool open = lo < hi && hi < n && sorted.row[hi - 1] == sorted.row[hi];
                if (open && head) hand_on(kCarryThrough);
                __syncthreads();
                if (open && !head) {
                    for (int w = me + 1; w < kOwnWarps; ++w) {
                        const int state = s_state[w];
                        if (state == kCarrySkip) continue;
#pragma unroll
                        for (int j = 0; j < N; ++j) acc[j] += s_carry[w * (32 * N) + e + j * 32];
                        if (state != kCarryThrough) break;
                    }
                    flush(sorted.row[hi - 1]);
                }
                if (stream) {
                    if (lo < hi && hi == n) writer.skip_to(n_rows * K);
                    writer.finish();
                }
                __syncthreads();
            }
            store = false;                   // what follows is added
            first += n;
        } while (first < last);
    });
}

// Calls f with the lanes per row that suit K floats.
template <int N>
struct Lanes { static constexpr int value = N; };
template <class F>
static int with_row_lanes(int K, F f) {
    const int words = (K + 3 + 3) / 4;
    if (words <= 2) return f(Lanes<2>{});
    if (words <= 4) return f(Lanes<4>{});
    if (words <= 8) return f(Lanes<8>{});
    if (words <= 16) return f(Lanes<16>{});
    return f(Lanes<32>{});
}

static int zero_rows(float* grad, int64_t n_floats, cudaStream_t stream) {
    SVOXB_CUDA(cudaMemsetAsync(grad, 0, (size_t)n_floats * sizeof(float), stream));
    return SVOXB_OK;
}

// Calls f with the columns per lane that suit K floats.
template <class F>
static int with_columns(int K, F f) {
    if (K <= 32) return f(Lanes<1>{});
    if (K <= 64) return f(Lanes<2>{});
    return f(Lanes<4>{});
}

static int launch_tiled(const int64_t* ids, const float* rows, int K, float* grad, TileLists t,
                        cudaStream_t stream) {
    int st;
    if ((st = keep_pool_cached())) return st;
    const int64_t Q = t.n_items;
    const size_t words = t.words();
    int32_t* mem = nullptr;
    SVOXB_CUDA(cudaMallocAsync((void**)&mem, (words + 2 * (size_t)Q) * sizeof(int32_t), stream));
    t.place_in(mem);
    int2* pair = reinterpret_cast<int2*>(mem + words);
    st = [&] {
        SVOXB_CUDA(cudaMemsetAsync(mem, 0, t.zero_words() * sizeof(int32_t), stream));
        const int sms = sm_count();
        auto grid_of = [&](auto kernel, int block, size_t smem, int64_t need, unsigned* grid) {
            int per_sm = 0;
            const int s2 = blocks_per_sm(reinterpret_cast<const void*>(kernel), block, smem, &per_sm);
            const int64_t most = (int64_t)sms * per_sm;
            *grid = (unsigned)(need < most ? need : most);
            return s2;
        };
        auto blocks = [&](int each) { return (Q + kPlaceBlock * each - 1) / (kPlaceBlock * each); };
        unsigned grid = 1;
        int s2;
        size_t smem = stepped(t.n_ranges, 2048) * sizeof(int32_t);
        if ((s2 = grid_of(count_ranges_kernel, kPlaceBlock, smem, blocks(4), &grid)))
            return s2;
        count_ranges_kernel<<<grid, kPlaceBlock, smem, stream>>>(ids, t);
        smem = stepped(t.max_tiles, 2048) * sizeof(int32_t);
        if ((s2 = grid_of(count_tiles_kernel, kPlaceBlock, smem, blocks(4), &grid))) return s2;
        count_tiles_kernel<<<grid, kPlaceBlock, smem, stream>>>(ids, t);
        if ((s2 = grid_of(place_tiles_kernel, kPlaceBlock, smem, blocks(kPlaceEach), &grid)))
            return s2;
        place_tiles_kernel<<<grid, kPlaceBlock, smem, stream>>>(ids, t, pair, K, grad);
        return with_columns(K, [&](auto columns) {
            auto own = own_rows_kernel<decltype(columns)::value>;
            const size_t bytes = TileSort::kBytes +
                                 kOwnWarps * (2 * 16 * kStageWords + 8 * StreamWriter::kPiece);
            const int s3 = grid_of(own, kOwnBlock, bytes, (int64_t)t.max_tiles + Q / kOwnItems, &grid);
            if (s3) return s3;
            own<<<grid, kOwnBlock, bytes, stream>>>(rows, (uint32_t)(Q - 1), K, grad, t, pair);
            SVOXB_CUDA(cudaGetLastError());
            return (int)SVOXB_OK;
        });
    }();
    cudaFreeAsync(mem, stream);
    return st;
}

// Which of the two a large gradient takes.  Summing by tiles writes the gradient once, and costs
// instructions per row of points (69 for 49 floats); adding bin by bin clears and adds in the L2, and
// costs a reduction per 16 bytes, which eight lanes share for rows of up to 29 floats and sixteen from
// there on.  So tiles need long rows, and points that fall on many different rows; the fewer points
// per row and the larger the gradient, the shorter rows may be.  Measured (us, bins / tiles; points
// spread over 7/8 of the rows, then 93 % of them in 3 % of the rows, as uniform points in a tree of
// coarse and fine leaves, then around one place, +- 8 % of the rows):
//
//   floats, MB   0.26 points a row            0.5                          1                           2
//   24, 1130     594/527  429/470  486/503    773/754  610/600  643/684    1116/1203 937/906 950/1023  1633/1873 1472/1476 1464/1604
//   28,  400     224/199  170/208  188/248    282/277  222/235  243/295    390/423   317/331 322/393   549/617   495/513   483/558
//   28,  800     435/347  304/329  350/365    538/485  414/415  451/485    758/783   629/586 641/668   1089/1184 991/970   973/1064
//   28, 2050     1067/822 740/771  850/795    1339/1176 1056/986 1123/1090 1920/1885 1604/1455 1645/1612  2888/3076 2532/2529 2539/2710
//   32,  400     200/194  190/176  183/243    248/267  244/213  234/284    358/381   357/289 342/351   579/558   586/442   554/501
//   32, 1130     530/436  438/412  436/444    654/637  623/516  587/587    973/988   987/728 901/829   1600/1475 1626/1157 1497/1286
//   49,  256     135/132  133/167  129/173    179/149  155/193  157/193    230/195   209/284 213/233   335/326   319/350   312/305
//   49,  400     211/180  178/196  178/188    261/215  217/228  220/242    339/292   303/285 302/301   502/474   476/415   459/437
//   49, 1130     585/385  385/412  434/413    692/487  520/518  548/501    879/746   805/663 789/692   1383/1131 1312/1049 1260/1082
//   76,  400     218/157  183/238  183/212    266/187  222/239  226/243    359/243   313/269 311/286   510/415   496/365   477/382
//  200,  400     184/151  188/209  166/156    244/175  238/208  228/202    328/227   292/252 290/292   462/317   402/413   410/415
//  200,  800     371/251  310/271  304/273    475/307  370/331  385/367    639/409   492/462 529/496   885/603   753/599   779/645
//  300,  400     189/156  222/265  175/185    271/189  227/260  224/242    357/242   305/338 309/352   500/333   424/453   431/462
//
// Around one place of +- 2 % tiles of up to 128 floats take at most 1.4 times as long as bins (400 MB, 0.26
// points a row, 162 / 207), longer rows, which do not fit a warp's registers at once, more below 768 MB
// (200 floats, 400 MB, 196 / 363; 2 GB 753 / 728).
static bool sums_by_tiles(int64_t n_slots, int K, int64_t Q) {
    const int64_t mb = n_slots * K >> 18;
    if (K <= 24) return false;
    if (K <= 29) return mb >= 768 && Q <= n_slots;
    if (K <= 32) return mb >= 768;
    return mb >= (K <= 128 || Q >= n_slots ? 384 : 768);
}

static int launch_scatter(const svoxb_tree* tree, const int64_t* ids, int64_t Q, const float* rows,
                          int K, float* grad, bool zero_first, cudaStream_t stream) {
    const int64_t n_slots = tree->M * tree->N * tree->N * tree->N, n_floats = n_slots * K;
    // Binned where the gradient outgrows the L2 and a good part of its records is touched (at
    // least every eighth or so, with 8 * 16 bytes of sorting against 260 of every row).
    const bool binned = zero_first && n_floats * 4 >= (96LL << 20) && Q >= n_slots / 4 &&
                        Q < (1LL << 31) - kBinRows && n_slots < (1LL << 31) &&
                        reinterpret_cast<uintptr_t>(grad) % 16 == 0;
    int st;
    if (binned && sums_by_tiles(n_slots, K, Q)) {
        const TileLists t(n_slots, Q, sm_count());
        if (t.max_tiles <= kMaxTiles) return launch_tiled(ids, rows, K, grad, t, stream);
    }
    if (!binned) {
        if (zero_first && (st = zero_rows(grad, n_floats, stream))) return st;
        if (Q == 0) return SVOXB_OK;
        const int64_t grid = (Q + kQueryBlock - 1) / kQueryBlock;
        if (grid > 0x7fffffffLL) return SVOXB_ERR_TOO_LARGE;
        return with_row_lanes(K, [&](auto lanes) {
            scatter_rows_kernel<decltype(lanes)::value><<<(unsigned)grid, kQueryBlock, 0, stream>>>(
                ids, Q, rows, K, grad, n_slots);
            SVOXB_CUDA(cudaGetLastError());
            return (int)SVOXB_OK;
        });
    }
    if ((st = keep_pool_cached())) return st;
    RowBins b{};
    b.shift = 2;                          // a bin is a whole number of 16-byte words
    while ((2LL << b.shift) * K * 4 <= ((int64_t)kReplayBinMB << 20)) ++b.shift;
    while (((n_slots - 1) >> b.shift) + 1 > kMaxBins) ++b.shift;
    b.n_bins = (int)(((n_slots - 1) >> b.shift) + 1);
    constexpr int kHead = 3 * kMaxBins + 32;
    int32_t* mem = nullptr;
    SVOXB_CUDA(cudaMallocAsync((void**)&mem, (kHead + 2 * (size_t)Q) * sizeof(int32_t), stream));
    b.count = mem;
    b.cursor = mem + kMaxBins;
    b.units = UnitCounters{mem + 3 * kMaxBins, mem + 3 * kMaxBins + 1, mem + 2 * kMaxBins};
    b.pair = reinterpret_cast<int2*>(mem + kHead);
    st = [&] {
        SVOXB_CUDA(cudaMemsetAsync(mem, 0, kHead * sizeof(int32_t), stream));
        const int sms = sm_count();
        int64_t grid = (Q + 256 * 16 - 1) / (256 * 16);
        if (grid > 8LL * sms) grid = 8LL * sms;
        count_rows_kernel<<<(unsigned)grid, 256, 0, stream>>>(ids, Q, n_slots, b);
        grid = (Q + kBinRows - 1) / kBinRows;
        if (grid > 8LL * sms) grid = 8LL * sms;
        place_rows_kernel<<<(unsigned)grid, 256, 0, stream>>>(ids, Q, n_slots, b);
        SVOXB_CUDA(cudaGetLastError());
        return with_row_lanes(K, [&](auto lanes) {
            auto k = scatter_binned_rows_kernel<decltype(lanes)::value>;
            int per_sm = 0;
            const int s2 = blocks_per_sm(reinterpret_cast<const void*>(k), kQueryBlock, 0, &per_sm);
            if (s2) return s2;
            const int blocks = sms * per_sm;
            // rows a warp takes per unit: the grid's window stays below a bin
            int64_t per_warp = Q / b.n_bins / ((int64_t)blocks * kQueryBlock);
            per_warp = per_warp < 1 ? 1 : per_warp > 4 ? 4 : per_warp;
            k<<<(unsigned)blocks, kQueryBlock, 0, stream>>>(Q, rows, K, grad, n_slots, b,
                                                            (int)per_warp);
            SVOXB_CUDA(cudaGetLastError());
            return (int)SVOXB_OK;
        });
    }();
    cudaFreeAsync(mem, stream);
    return st;
}

// The same from the points themselves.
static int launch_query_backward(const svoxb_tree* tree, const float* indices, int64_t Q,
                                 const float* rows, int K, float* grad, bool zero_first,
                                 cudaStream_t stream) {
    if (Q == 0) return launch_scatter(tree, nullptr, 0, rows, K, grad, zero_first, stream);
    int st = keep_pool_cached();
    if (st) return st;
    int64_t* ids = nullptr;
    SVOXB_CUDA(cudaMallocAsync((void**)&ids, (size_t)Q * sizeof(int64_t), stream));
    st = launch_query(tree, indices, Q, nullptr, ids, nullptr, nullptr, 0, stream);
    if (st == SVOXB_OK) st = launch_scatter(tree, ids, Q, rows, K, grad, zero_first, stream);
    cudaFreeAsync(ids, stream);
    return st;
}

}  // namespace svoxb
