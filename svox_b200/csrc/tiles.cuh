// Adding many rows into a large buffer (a gradient) whose rows are hit in any order, without a
// single reduction in the common case: the items are sorted by TILE, a range of some thousand rows
// of the buffer, one block takes a tile, sorts its items by row in shared memory, sums every row's
// items in registers and writes the row once, zeros where it has none.
//
// Clearing the buffer and adding with red.global moves every row through the L2 once per item and
// once for the zeros, and the L2 takes 46 G reductions of a 112-byte row a second (5.2 TB/s, measured
// with all of them hits); here the buffer is written once and only the items are read.
//
//   count    items per tile
//   scan     where each tile's items begin; tiles with very many items (HOT) become several units
//   place    the items' references, tile by tile; hot tiles are cleared
//   own      (the caller's kernel) a block per unit, through TileSort
#pragma once

#include "common.cuh"

namespace svoxb {

constexpr int kOwnBlock = 512;
constexpr int kOwnWarps = kOwnBlock / 32;
constexpr int kOwnItems = 4096;                // items a block sorts at a time
constexpr int kHotItems = 8 * kOwnItems;       // a tile with more is shared out, see scan_tiles_kernel
constexpr int kMinTileShift = 6;
// Tiles up to which a block counts in shared memory.
constexpr int kMaxSharedTiles = 12288;

// Lists of items by tile, in one allocation.
struct TileLists {
    int32_t* head;       // [0] next unit  [1] hot units  [2] hot tiles
    int32_t* count;      // [n_tiles] items of a tile
    int32_t* end;        // [n_tiles] end of those placed so far; after `place` of all
    int2* hot_unit;      // {tile, first item within the tile}
    int32_t* hot_tile;
    int shift;           // log2 of a tile's rows
    int n_tiles;
    int64_t n_rows;

    // Hot units and tiles that `items` items can make.
    static int64_t most_hot(int64_t items) { return items / kOwnItems * 5 / 4 + 2; }
    static size_t words(int n_tiles, int64_t items) {
        return (32 + 2 * (size_t)n_tiles + 3 + 3 * (size_t)most_hot(items)) & ~(size_t)1;
    }
    // Words that are zero before `count`.
    size_t zero_words() const { return 32 + (size_t)n_tiles; }
    void place_in(int32_t* mem, int64_t items) {
        head = mem;
        count = mem + 32;
        end = count + n_tiles;
        hot_unit = reinterpret_cast<int2*>(mem + ((32 + 2 * (size_t)n_tiles + 1) & ~(size_t)1));
        hot_tile = reinterpret_cast<int32_t*>(hot_unit + most_hot(items));
    }
};

// One block.  A tile's items are one unit of work, unless there are more than kHotItems of them
// (rows that very many items hit: the leaf that a camera stands in): then every kOwnItems of them
// are, so that the device shares in them, and what they add goes into a cleared tile.
__global__ void __launch_bounds__(1024) scan_tiles_kernel(TileLists t) {
    __shared__ int s_sum[32];
    __shared__ int s_carry;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) s_carry = 0;
    __syncthreads();
    for (int base = 0; base < t.n_tiles; base += 1024) {
        const int i = base + tid;
        const int n = i < t.n_tiles ? t.count[i] : 0;
        int x = n;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) s_sum[tid >> 5] = x;
        __syncthreads();
        if (tid < 32) {
            int w = s_sum[tid];
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const int y = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += y;
            }
            s_sum[tid] = w;
        }
        __syncthreads();
        const int first = s_carry + (tid >= 32 ? s_sum[(tid >> 5) - 1] : 0) + x - n;
        if (i < t.n_tiles) {
            t.end[i] = first;
            if (n > kHotItems) {
                const int units = (n + kOwnItems - 1) / kOwnItems;
                const int at = atomicAdd(t.head + 1, units);
                for (int u = 0; u < units; ++u) t.hot_unit[at + u] = make_int2(i, u * kOwnItems);
                t.hot_tile[atomicAdd(t.head + 2, 1)] = i;
            }
        }
        __syncthreads();
        if (tid == 0) s_carry += s_sum[31];
        __syncthreads();
    }
}

// Clears the rows of the hot tiles; all threads of the grid.
__device__ __forceinline__ void clear_hot_tiles(const TileLists& t, int K, float* __restrict__ out) {
    const int n = *(volatile int32_t*)(t.head + 2);
    for (int h = 0; h < n; ++h) {
        const int64_t first = (int64_t)t.hot_tile[h] << t.shift;
        const int64_t left = t.n_rows - first, rows = (int64_t)1 << t.shift;
        float* __restrict__ to = out + first * K;
        const int64_t floats = (left < rows ? left : rows) * K;
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < floats;
             i += (int64_t)gridDim.x * blockDim.x)
            to[i] = 0.f;
    }
}

// Shared memory of a block: end of each row's items (two 16-bit numbers per word; an item count
// fits, kOwnItems < 2^16), and the items row by row with their rows.
struct TileSort {
    uint32_t* end;
    uint32_t* item;
    uint16_t* row;

    static __host__ __device__ size_t bytes(int shift) {
        return ((size_t)2 << shift) + (size_t)kOwnItems * 6;
    }
    __device__ __forceinline__ explicit TileSort(unsigned char* smem, int shift) {
        end = reinterpret_cast<uint32_t*>(smem);
        item = end + (1 << (shift - 1));
        row = reinterpret_cast<uint16_t*>(item + kOwnItems);
    }
    // Number of the items in rows up to `r` of the tile.
    __device__ __forceinline__ int upto(int r) const {
        return r < 0 ? 0 : reinterpret_cast<const uint16_t*>(end)[r];
    }
    // Sorts n <= kOwnItems items, `get(i)` = {row within the tile, item}, by row.  All threads;
    // ends with a barrier.
    template <class Get>
    __device__ __forceinline__ void sort(int n, int shift, Get get) const {
        __shared__ int s_sum[kOwnWarps];
        const int tid = threadIdx.x, lane = tid & 31;
        const int words = 1 << (shift - 1);
        for (int w = tid; w < words; w += kOwnBlock) end[w] = 0;
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < n; i += kOwnBlock) {
            const int r = get(i).x;
            atomicAdd(end + (r >> 1), 1u << (16 * (r & 1)));
        }
        __syncthreads();
        // words [tid * per, + per) of this thread: their sum, then exclusive sums in place
        const int per = words > kOwnBlock ? words / kOwnBlock : 1;
        int own = 0;
        if (tid * per < words)
            for (int w = 0; w < per; ++w) {
                const uint32_t c = end[tid * per + w];
                own += (int)(c & 0xffffu) + (int)(c >> 16);
            }
        int x = own;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) s_sum[tid >> 5] = x;
        __syncthreads();
        int run = x - own;
        for (int w = 0; w < (tid >> 5); ++w) run += s_sum[w];
        if (tid * per < words)
            for (int w = 0; w < per; ++w) {
                const uint32_t c = end[tid * per + w];
                const int lo = (int)(c & 0xffffu), hi = (int)(c >> 16);
                end[tid * per + w] = (uint32_t)run | ((uint32_t)(run + lo) << 16);
                run += lo + hi;
            }
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < n; i += kOwnBlock) {
            const int2 it = get(i);
            const int half = 16 * (it.x & 1);
            const int pos = (int)((atomicAdd(end + (it.x >> 1), 1u << half) >> half) & 0xffffu);
            item[pos] = (uint32_t)it.y;
            row[pos] = (uint16_t)it.x;
        }
        __syncthreads();
    }
    // Writes zeros to the rows [0, n_rows) of `out` that have no item.
    __device__ __forceinline__ void clear_empty(int n_rows, int K, float* __restrict__ out) const {
        const int lane = threadIdx.x & 31;
        const bool vec_ok = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
        for (int r0 = threadIdx.x & ~31; r0 < n_rows; r0 += kOwnBlock) {
            const int r = r0 + lane;
            unsigned none = __ballot_sync(0xffffffffu, r < n_rows && upto(r) == upto(r - 1));
            float* __restrict__ to = out + (int64_t)r0 * K;
            if (none == 0xffffffffu && vec_ok) {
                for (int i = lane; i < 8 * K; i += 32)
                    reinterpret_cast<float4*>(to)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
                for (; none != 0u; none &= none - 1u) {
                    float* __restrict__ at = to + (__ffs(none) - 1) * K;
                    for (int e = lane; e < K; e += 32) at[e] = 0.f;
                }
            }
        }
    }
};

// Writes a stretch of consecutive floats, appended row by row by a warp, in aligned pieces of
// 512 bytes: rows that begin and end inside 32-byte sectors reach DRAM at 2.9 TB/s when they are
// stored one by one (3.76 GB of 196-byte rows in 1.30 ms).
struct StreamWriter {
    static constexpr int kPiece = 128;              // floats
    float* buf;         // the warp's 2 * kPiece floats of shared memory, 16-byte aligned: the piece
                        // that `pos` lies in and the next one, zeros where nothing was put yet
    float* out;         // 16-byte aligned
    int start, pos;     // floats of `out`: first one of the stretch, next one

    __device__ __forceinline__ void clear() {
        float4* const b = reinterpret_cast<float4*>(buf) + (threadIdx.x & 31);
        b[0] = b[32] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
    }
    __device__ __forceinline__ void begin(float* to, int at) {
        out = to;
        start = pos = at;
    }
    // Writes the floats of the piece `pos` lies in from `start` on, up to `until`.
    __device__ __forceinline__ void write_some(float4 v, int until) {
        const int i = (pos & ~(kPiece - 1)) + 4 * (threadIdx.x & 31);
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + j >= start && i + j < until) out[i + j] = x[j];
    }
    // Writes the piece that `pos` lies in.
    __device__ __forceinline__ void drain() {
        __syncwarp();
        float4* const b = reinterpret_cast<float4*>(buf) + (threadIdx.x & 31);
        const float4 v = b[0];
        b[0] = b[32];
        b[32] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int piece = pos & ~(kPiece - 1);
        if (piece >= start) reinterpret_cast<float4*>(out + piece)[threadIdx.x & 31] = v;
        else write_some(v, piece + kPiece);
        __syncwarp();
    }
    // Zeros up to float `to`.
    __device__ __forceinline__ void skip_to(int to) {
        while (((to ^ pos) & ~(kPiece - 1)) != 0) {
            drain();
            pos = (pos | (kPiece - 1)) + 1;
        }
        pos = to;
    }
    // n <= min(kPiece, 32 * N) floats, lane e holds those at e, e + 32, ...
    template <int N>
    __device__ __forceinline__ void append(const float (&v)[N], int n) {
        const int e = threadIdx.x & 31;
        float* const to = buf + (pos & (kPiece - 1)) + e;
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (e + j * 32 < n) to[j * 32] = v[j];
        const int next = pos + n;
        if (((pos ^ next) & ~(kPiece - 1)) != 0) drain();
        pos = next;
    }
    __device__ __forceinline__ void finish() {
        __syncwarp();
        write_some(reinterpret_cast<const float4*>(buf)[threadIdx.x & 31], pos);
        __syncwarp();
        clear();
    }
};

// Where a run of equal rows crosses from one warp's range of sorted items to the next: the warp
// where it begins adds up what the others found of it.
enum { kCarryNone = 0, kCarryEnds = 1, kCarryThrough = 2, kCarrySkip = 3 };

// Units of a launch: hot units first, then the tiles that are not hot, handed out in order.
// `work(tile, first, last, hot)` by all threads, items [first, last) of the sorted list.
template <class Work>
__device__ __forceinline__ void owned_units(const TileLists& t, int lo_tile, int hi_tile, Work work) {
    __shared__ int s_unit;
    const int n_hot = *(volatile int32_t*)(t.head + 1);
    const int all = n_hot + hi_tile - lo_tile;
    int next = 0;
    if (threadIdx.x == 0) next = atomicAdd(t.head, 1);
    for (;;) {
        if (threadIdx.x == 0) s_unit = next;
        __syncthreads();
        const int u = s_unit;
        if (u >= all) break;
        if (threadIdx.x == 0) next = atomicAdd(t.head, 1);      // arrives during this unit
        int tile, from = 0;
        const bool hot = u < n_hot;
        if (hot) {
            const int2 h = t.hot_unit[u];
            tile = h.x;
            from = h.y;
        } else {
            tile = lo_tile + u - n_hot;
        }
        const int n = t.count[tile];
        const int first = t.end[tile] - n;
        if (hot) {
            if (tile >= lo_tile && tile < hi_tile)
                work(tile, first + from, first + (n < from + kOwnItems ? n : from + kOwnItems), true);
        } else if (n <= kHotItems) {
            work(tile, first, first + n, false);
        }
        __syncthreads();
    }
}

}  // namespace svoxb
