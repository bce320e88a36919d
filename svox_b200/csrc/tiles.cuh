// Adding many rows into a large buffer (a gradient) whose rows are hit in any order, without a
// single reduction in the common case: the items are sorted by TILE, a range of some thousand rows
// of the buffer, one block takes a tile, sorts its items by row in shared memory, sums every row's
// items in registers and writes the row once, zeros where it has none.
//
// Clearing the buffer and adding with red.global moves every row through the L2 once per item and
// once for the zeros, and the L2 takes 46 G reductions of a 112-byte row a second (5.2 TB/s, measured
// with all of them hits); here the buffer is written once and only the items are read.
//
// Items are spread unevenly: coarse leaves are hit more often than fine ones, points lie near a
// surface.  So the buffer is first divided into equal RANGES of 2^shift rows, and each is cut into 1,
// 2, 4 .. tiles, as many as bring a block no more than it can sort at a time.  (Cut by the average
// alone, 14.7 M uniform points into a 1024^3 tree of three shells, 56 M rows of 28 floats, made tiles of
// 33 000 items: 5.95 ms, now 2.22; 0.7 M points around one place of 400 MB of 76 floats: 0.84 -> 0.25.)
//
//   count    items per range; the last block cuts the ranges into tiles
//   recount  items per tile, if any range was cut; the last block lists where each tile's begin, and
//            the tiles that have very many all the same (HOT), which become several units of work
//   place    the items' references, tile by tile; hot tiles are cleared
//   own      (the caller's kernel) a block per unit, through TileSort
#pragma once

#include "common.cuh"

namespace svoxb {

constexpr int kOwnBlock = 512;
constexpr int kOwnWarps = kOwnBlock / 32;
// Items a block sorts at a time; with two blocks per SM there is room for 4840.  (4096 left half of the
// tiles of 2^24 uniform points in a 256^3 tree, 4096 +- 64 items each, a second turn for a few items:
// 2.07 ms, 2.00 with 4608 or 4800.)
constexpr int kOwnItems = 4800;
// A tile with more than kOwnItems is shared out, see list_tiles, if its rows have this many on
// average, or if it would take one block more than kHotTurns turns.
constexpr int kHotRow = 16, kHotTurns = 8;
constexpr int kMinTileShift = 6, kMaxTileShift = 12;
// Tiles that a block counts in shared memory; buffers that need more are not summed by tiles.
constexpr int kMaxTiles = 24576;

// Lists of items by tile, in one allocation.
struct TileLists {
    int32_t* head;       // [0] next unit  [1] hot units  [2] hot tiles  [3] tiles
                         // [4], [5] blocks that are done with counting, recounting
    int32_t* in_range;   // [n_ranges] items of a range
    int32_t* count;      // [max_tiles] items of a tile
    int32_t* end;        // [max_tiles] end of those placed so far; after `place` of all
    uint32_t* cut;       // [n_ranges] first tile; bits 28-31: log2 of the range's tiles
    uint32_t* where;     // [max_tiles] first row / 2^kMinTileShift; bits 28-31: log2 of the tile's
                         // rows, less kMinTileShift
    int2* hot_unit;      // {tile, first item within the tile}
    int32_t* hot_tile;
    int shift;           // log2 of a range's rows
    int n_ranges, max_tiles;
    int64_t n_rows, n_items;

    static constexpr size_t up4(size_t n) { return (n + 3) & ~(size_t)3; }
    // Hot units and tiles that the items can make.
    int64_t most_hot() const { return 2 * n_items / kOwnItems + 2; }
    // Words that are zero before `count`.
    size_t zero_words() const { return 32 + up4(n_ranges) + up4(max_tiles); }
    size_t words() const {
        return zero_words() + 2 * up4(max_tiles) + up4(n_ranges) + up4(3 * (size_t)most_hot());
    }
    // Ranges have 2^kMaxTileShift rows, or fewer where the `sms` processors would not come to about two
    // rounds of two blocks each with them: 0.5 M points into 1.05 M rows of 100 floats (256 ranges of
    // 4096 rows) 295 us, 190 with 1024 ranges; 0.1 M into 0.21 M rows of 1000 floats 1254, 314; 0.5 M
    // into 2.05 M of 128 (500 ranges) 424, 290.  From there on more ranges cost more than they gain (0.6 M
    // into 2.4 M of 49: 585 ranges 178, 1170 ranges 192).
    TileLists(int64_t rows, int64_t items, int sms) : n_rows(rows), n_items(items) {
        shift = kMaxTileShift;
        while (shift > kMinTileShift && (rows >> shift) < 4 * (int64_t)sms - sms / 4) --shift;
        n_ranges = (int)(((rows - 1) >> shift) + 1);
        // A range is cut into 2^n tiles, n > 0, only with more than 2^(n-1) * kOwnItems items.
        const int64_t most = n_ranges + 2 * items / kOwnItems + 1;
        max_tiles = most < INT32_MAX ? (int)most : INT32_MAX;
    }
    void place_in(int32_t* mem) {
        head = mem;
        in_range = mem + 32;
        count = in_range + up4(n_ranges);
        end = count + up4(max_tiles);
        where = reinterpret_cast<uint32_t*>(end + up4(max_tiles));
        cut = where + up4(max_tiles);
        hot_unit = reinterpret_cast<int2*>(cut + up4(n_ranges));
        hot_tile = reinterpret_cast<int32_t*>(hot_unit + most_hot());
    }
    // Tile of a row.
    __device__ __forceinline__ int tile_of(int64_t row) const {
        const uint32_t c = __ldg(cut + (row >> shift));
        return (int)(c & 0x0fffffffu) +
               (int)(((uint32_t)row & ((1u << shift) - 1u)) >> (shift - (int)(c >> 28)));
    }
    __device__ __forceinline__ bool is_hot(int tile, int items) const {
        return items > kOwnItems &&
               (items > kHotTurns * kOwnItems || items >= kHotRow << tile_shift(tile));
    }
    __device__ __forceinline__ int64_t first_row(int tile) const {
        return (int64_t)(where[tile] & 0x0fffffffu) << kMinTileShift;
    }
    __device__ __forceinline__ int tile_shift(int tile) const {
        return (int)(where[tile] >> 28) + kMinTileShift;
    }
};

// Sum of n over the threads before this one; *total: over all.  `s_sum`: BLOCK / 32 words.
template <int BLOCK>
__device__ __forceinline__ int sum_before(int n, int* s_sum, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = n;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_sum[warp] = x;
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < BLOCK / 32; ++w) {
        const int v = s_sum[w];
        if (w < warp) before += v;
        all += v;
    }
    __syncthreads();
    *total = all;
    return before + x - n;
}

// Whether this block is the last one of the grid to come here; it then sees what the others wrote
// before.  All threads.
__device__ __forceinline__ bool last_block(int32_t* done) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// Lists where the tiles' items begin; one block.  A tile's items are one unit of work, unless it is
// HOT: then every kOwnItems of them are, so that the device shares in them, and what they add goes
// into a cleared tile.  With many items per row (the leaf that a camera stands in) the reductions for
// that are few; else it is the lesser evil.  `counted`: items per tile.
template <int BLOCK>
__device__ __forceinline__ void list_tiles(const TileLists& t, const int32_t* counted) {
    __shared__ int s_sum[BLOCK / 32];
    const int n_tiles = t.head[3];
    int run = 0;
    for (int base = 0; base < n_tiles; base += 4 * BLOCK) {
        const int i = base + 4 * (int)threadIdx.x;
        int n[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) n[j] = i + j < n_tiles ? __ldcg(counted + i + j) : 0;
        int total;
        int first = run + sum_before<BLOCK>(n[0] + n[1] + n[2] + n[3], s_sum, &total);
        run += total;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i + j >= n_tiles) break;
            if (counted != t.count) t.count[i + j] = n[j];
            t.end[i + j] = first;
            first += n[j];
            if (!t.is_hot(i + j, n[j])) continue;
            const int units = (n[j] + kOwnItems - 1) / kOwnItems;
            const int at = atomicAdd(t.head + 1, units);
            for (int u = 0; u < units; ++u) t.hot_unit[at + u] = make_int2(i + j, u * kOwnItems);
            t.hot_tile[atomicAdd(t.head + 2, 1)] = i + j;
        }
    }
}

// Cuts the ranges into tiles, and lists these if they are the ranges; one block.
template <int BLOCK>
__device__ __forceinline__ void cut_ranges(const TileLists& t) {
    __shared__ int s_sum[BLOCK / 32];
    int run = 0;
    for (int base = 0; base < t.n_ranges; base += BLOCK) {
        const int r = base + (int)threadIdx.x;
        int levels = 0;
        if (r < t.n_ranges) {
            const int64_t items = __ldcg(t.in_range + r);
            while (levels < t.shift - kMinTileShift && items > (int64_t)kOwnItems << levels) ++levels;
        }
        int total;
        const int first = run + sum_before<BLOCK>(r < t.n_ranges ? 1 << levels : 0, s_sum, &total);
        run += total;
        if (r < t.n_ranges) {
            t.cut[r] = (uint32_t)first | (uint32_t)levels << 28;
            const int shift = t.shift - levels;
            const uint32_t row0 = (uint32_t)(((int64_t)r << t.shift) >> kMinTileShift);
            for (int j = 0; j < 1 << levels; ++j)
                t.where[first + j] = (row0 + ((uint32_t)j << (shift - kMinTileShift))) |
                                     (uint32_t)(shift - kMinTileShift) << 28;
        }
    }
    if (threadIdx.x == 0) t.head[3] = run;
    __syncthreads();
    if (run == t.n_ranges) list_tiles<BLOCK>(t, t.in_range);
}

// Clears the rows of the hot tiles; all blocks of the grid.
__device__ __forceinline__ void clear_hot_tiles(const TileLists& t, int K, float* __restrict__ out) {
    const int n = t.head[2];
    for (int h = blockIdx.x; h < n; h += gridDim.x) {
        const int64_t first = t.first_row(t.hot_tile[h]);
        const int64_t left = t.n_rows - first, rows = (int64_t)1 << t.tile_shift(t.hot_tile[h]);
        float* __restrict__ to = out + first * K;
        const int64_t floats = (left < rows ? left : rows) * K;
        for (int64_t i = threadIdx.x; i < floats; i += blockDim.x) to[i] = 0.f;
    }
}

// Shared memory of a block: end of each row's items (two 16-bit numbers per word; an item count
// fits, kOwnItems < 2^16), and the items row by row with their rows.
struct TileSort {
    uint32_t* end;
    uint32_t* item;
    uint16_t* row;

    static constexpr size_t kBytes = ((size_t)2 << kMaxTileShift) + (size_t)kOwnItems * 6;
    __device__ __forceinline__ explicit TileSort(unsigned char* smem) {
        end = reinterpret_cast<uint32_t*>(smem);
        item = end + (1 << (kMaxTileShift - 1));
        row = reinterpret_cast<uint16_t*>(item + kOwnItems);
    }
    // Number of the items in rows up to `r` of the tile.
    __device__ __forceinline__ int upto(int r) const {
        return r < 0 ? 0 : reinterpret_cast<const uint16_t*>(end)[r];
    }
    // Sorts n <= kOwnItems items, `get(i)` = {row within the tile, item}, by row of a tile of 2^shift.
    // All threads; ends with a barrier.
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
    // Writes zeros to the rows [0, n_rows) of `out`, 16-byte aligned, that have no item.
    __device__ __forceinline__ void clear_empty(int n_rows, int K, float* __restrict__ out) const {
        const int lane = threadIdx.x & 31;
        for (int r0 = threadIdx.x & ~31; r0 < n_rows; r0 += kOwnBlock) {
            const int r = r0 + lane;
            unsigned none = __ballot_sync(0xffffffffu, r < n_rows && upto(r) == upto(r - 1));
            float* __restrict__ to = out + (int64_t)r0 * K;
            if (none == 0xffffffffu) {
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
__device__ __forceinline__ void owned_units(const TileLists& t, Work work) {
    __shared__ int s_unit;
    const int n_hot = *(volatile int32_t*)(t.head + 1);
    const int all = n_hot + *(volatile int32_t*)(t.head + 3);
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
            tile = u - n_hot;
        }
        const int n = t.count[tile];
        const int first = t.end[tile] - n;
        if (hot) {
            work(tile, first + from, first + (n < from + kOwnItems ? n : from + kOwnItems), true);
        } else if (!t.is_hot(tile, n)) {
            work(tile, first, first + n, false);
        }
        __syncthreads();
    }
}

}  // namespace svoxb
