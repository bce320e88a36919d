// The render index of an octree (N = 2): what a march reads instead of walking `child` from
// the root and fetching every leaf's density from its 100- to 300-byte record.
//
// Level L of the tree is a dense TABLE of 2^L cells per side; a table cell that holds a node
// gets a BRICK, the 8x8x8 grid of the three levels below it.  Both consist of one ENTRY of two
// words per cell, z fastest:
//   word 0   0x00000001 .. 0x7f800000   the cell lies in a leaf that passes the density test;
//                                       the word is its density (softplus applied)
//            kWordEmpty                 in a leaf that fails it
//            kWordFetch                 passes it, but the density is no positive float
//                                       (possible below a negative threshold only)
//            kWordWalk                  the tree goes deeper here: walk `child`
//            negative (table only)      kWordBrick | brick id
//   word 1   bits 28-31: the leaf's depth; bits 0-27: its slot.  kWordWalk: the node to walk on
//            from, in bits 28-31 the depth of its children, or 0: walk from the root.  (Trees
//            of 34 M nodes or more, which get no bricks, and cells beyond the last brick;
//            200 000 rays through 34.2 M nodes: 9.2 ms if all walk from the root.)
// so that one 8-byte load per sample brings all that the march needs of a leaf.
//
// Built per call (`data` can change between any two): one thread per table cell, then one per
// brick cell.  The bound is the 64 bytes that DRAM delivers for every leaf's density (530 MB for
// the 8.3 M leaves of a 512^3 shell).
#pragma once

#include "query.cuh"

namespace svoxb {

// Whether an item log (render_queue.cuh) can be replayed: the forward did not ask for more chunks
// than it holds (word 0), and did not give the log up (word kLogGivenUp).
constexpr int kLogGivenUp = 4;
__device__ __forceinline__ bool log_complete(const int32_t* log, int64_t capacity) {
    return (int64_t)log[0] <= capacity && log[kLogGivenUp] == 0;
}

// A launch that is a FALLBACK for a log that cannot be replayed: its kernels do their work only
// in that case, so the host can enqueue replay and fallback without knowing which of the two
// applies.  `log` null: unconditional.
struct LogGate {
    const int32_t* log = nullptr;
    int64_t capacity = 0;
    __device__ __forceinline__ bool closed() const {
        return log != nullptr && log_complete(log, capacity);
    }
};

constexpr int kBrickLevels = 3;
constexpr int kBrickCells = 512;
constexpr int64_t kMaxPlace = 1 << 28;       // word 1 has 28 bits for a slot or a node
constexpr int64_t kIndexMaxNodes = kMaxPlace / 8;   // a tree with more nodes gets no bricks
constexpr int kMaxBricks = 1 << 17;
constexpr int kMaxTableLevel = 7;
constexpr int kPosBits = 23;                 // position bits below the binary point, see march

constexpr int32_t kWordInf = 0x7f800000;
constexpr int32_t kWordEmpty = kWordInf + 1;
constexpr int32_t kWordFetch = kWordInf + 2;   // these two leave the march's ordinary route
constexpr int32_t kWordWalk = kWordInf + 3;
constexpr int32_t kWordBrick = INT32_MIN;

__device__ __forceinline__ float sigmoid_ref(float x) { return 1 / (1 + expf(-x)); }
__device__ __forceinline__ float softplus_m1(float x) { return logf(1 + expf(x - 1)); }

// The index as the march sees it: one buffer of entries.
struct TreeIndex {
    const int2* table = nullptr;      // (2^level)^3 entries, z fastest, at the start
    uint32_t bricks = 0;              // from this entry on: kBrickCells per brick
    int level = 0;
    // What a march needs of the level, worked out here once: a number whose last place is the side
    // of a brick's cell, the place of a table cell among such cells, and the table's row length.
    float fine = 0.f;
    uint32_t cell_mask = 0, row = 0;

    static TreeIndex at(const int2* table, uint32_t bricks, int level) {
        const int finest = level + kBrickLevels;
        return TreeIndex{table, bricks, level, (float)(1 << (kPosBits - finest)),
                         ((1u << level) - 1u) << kBrickLevels, 1u << level};
    }
};

// One density out of its record.  Without the 64-byte hint the L2 fetched 128 bytes for each of
// these scattered sectors.
__device__ __forceinline__ float ld_density(const float* a) {
    float v;
    asm("ld.global.nc.L2::64B.f32 %0, [%1];" : "=f"(v) : "l"(a));
    return v;
}

__device__ __forceinline__ int32_t leaf_word(float raw, float thresh, int softplus) {
    const float sigma = softplus ? softplus_m1(raw) : raw;
    if (!(sigma > thresh)) return kWordEmpty;
    const int32_t bits = __float_as_int(sigma);
    return bits > 0 ? bits : kWordFetch;
}
__device__ __forceinline__ int32_t leaf_place(int depth, int64_t slot) {
    return (int32_t)(((uint32_t)depth << 28) | (uint32_t)slot);
}

__global__ void __launch_bounds__(256)
build_table_kernel(const int32_t* __restrict__ child, const float* __restrict__ data, int K,
                   int64_t M, int L, float thresh, int softplus, int brick_cap,
                   int2* __restrict__ table, int32_t* __restrict__ counter,
                   int32_t* __restrict__ roots, const uint8_t* __restrict__ marks, LogGate gate) {
    if (gate.closed()) return;
    const int S = (1 << L) - 1;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (1 << (3 * L));
         idx += gridDim.x * blockDim.x) {
        const int iz = idx & S, iy = (idx >> L) & S, ix = idx >> (2 * L);
        int64_t node = 0;
        int2 entry = make_int2(kWordWalk, 0);
        for (int l = 0; l < L; ++l) {
            const int b = L - 1 - l;
            const int64_t slot = node * 8 + ((((ix >> b) & 1) << 2) | (((iy >> b) & 1) << 1) |
                                             ((iz >> b) & 1));
            const int32_t e = __ldg(child + slot);
            if (e == 0) {
                const int32_t word = leaf_word(ld_density(data + slot * K + (K - 1)), thresh, softplus);
                if (slot < kMaxPlace) entry = make_int2(word, leaf_place(l + 1, slot));
                break;
            }
            node += e;
            if (node < 0 || node >= M) break;             // corrupt: reported by the march
            if (b != 0) continue;
            // without a brick the march walks on from the node
            if (node < kMaxPlace) entry.y = leaf_place(L + 1, node);
            if (brick_cap > 0 && (marks == nullptr || marks[idx] != 0)) {
                const int id = atomicAdd(counter, 1);
                if (id < brick_cap) {
                    roots[id] = (int32_t)node;
                    entry.x = kWordBrick | id;
                }
            }
        }
        table[idx] = entry;
    }
}

// One thread per brick cell: the loads on the way down are shared by a warp's neighbouring cells,
// the stores run through a brick.  (With one thread per 2x2x2 group and eight loads in flight each
// the kernel took 183 us instead of 114 on the 512^3 shell, 980 instead of 619 on 1024^3 shells.)
__global__ void __launch_bounds__(256)
fill_bricks_kernel(const int32_t* __restrict__ child, const float* __restrict__ data, int K,
                   int64_t M, int L, float thresh, int softplus, int cap,
                   int32_t* __restrict__ counter, const int32_t* __restrict__ roots,
                   int2* __restrict__ bricks, LogGate gate) {
    if (gate.closed()) return;
    int n = *(volatile int32_t*)counter;
    if (n > cap) n = cap;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)n * kBrickCells;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i & (kBrickCells - 1));
        const int x = c >> 6, y = (c >> 3) & 7, z = c & 7;
        int64_t node = __ldg(roots + (i >> 9));
        int2 entry = make_int2(kWordWalk, 0);
#pragma unroll
        for (int l = 1; l <= kBrickLevels; ++l) {
            const int b = kBrickLevels - l;
            const int64_t slot = node * 8 + ((((x >> b) & 1) << 2) | (((y >> b) & 1) << 1) |
                                             ((z >> b) & 1));
            const int32_t e = __ldg(child + slot);
            if (e == 0) {
                entry = make_int2(leaf_word(ld_density(data + slot * K + (K - 1)), thresh, softplus),
                                  leaf_place(L + l, slot));
                break;
            }
            if (l == kBrickLevels) entry.y = leaf_place(L + l, node);   // the tree goes deeper
            node += e;
            if (node < 0 || node >= M) break;              // corrupt: reported by the march
        }
        bricks[i] = entry;
    }
    if (gate.log != nullptr) {
        // counter[1]: blocks that have read the count; the last one clears both for the next build
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(counter + 1, 1) == (int)gridDim.x - 1) counter[0] = counter[1] = 0;
        }
    }
}

// Grid of an index-building kernel over n items: enough blocks to fill the device, not one
// per 256 items.
inline unsigned index_grid(int64_t n, int block, int sms) {
    const int64_t need = (n + block - 1) / block, most = (int64_t)sms * (2048 / block) * 2;
    return (unsigned)(need < most ? (need > 0 ? need : 1) : most);
}

// Where the parts of the index lie in its buffer (int32 words, 128-byte aligned parts):
// table | brick counter | brick roots | bricks.
struct IndexLayout {
    int level = 0, cap = 0;
    int64_t cells = 0;
    size_t counter = 0, roots = 0, bricks = 0, words = 0;

    // A complete tree (all leaves at one depth) that fits the largest table gets the table at
    // its leaves' level: no bricks, which would hold every leaf 8 or 64 times.  Any other
    // gets it at the deepest level whose complete tree its nodes could hold, at most 6 (64^3
    // cells, 1 MB), or 7 for trees of several million nodes, whose leaves lie up to ten levels
    // deep: the bricks then still reach them.
    static IndexLayout of(int64_t M, int max_bricks) {
        IndexLayout l;
        int full = 0;                    // deepest level of a complete tree of at most M nodes
        int64_t have = 1, pw = 1;
        while (full < kMaxTableLevel && have + 8 * pw <= M) {
            pw *= 8;
            have += pw;
            ++full;
        }
        const bool complete = have == M && full < kMaxTableLevel;
        const int most = M >= (4LL << 20) ? 7 : 6;
        l.level = complete ? full + 1 : full < most ? full : most;
        if (l.level < 1) l.level = 1;
        l.cells = (int64_t)1 << (3 * l.level);
        if (!complete && M < kIndexMaxNodes) {
            l.cap = (int)(l.cells < M ? l.cells : M);
            if (l.cap > max_bricks) l.cap = max_bricks;
        }
        auto up = [](size_t w) { return (w + 31) & ~(size_t)31; };
        l.counter = up(2 * (size_t)l.cells);
        l.roots = l.counter + 32;
        l.bricks = up(l.roots + (size_t)l.cap);
        l.words = l.bricks + (size_t)l.cap * (2 * kBrickCells);
        return l;
    }
    // The same with as many bricks as `room` words hold, at most max_bricks; `words` > room: there
    // is not even room for the table.
    static IndexLayout within(int64_t M, int max_bricks, int64_t room) {
        const int64_t left = room - (int64_t)of(M, 0).words - 64;
        const int64_t bricks = left / (2 * kBrickCells + 1);
        return of(M, bricks < 0 ? 0 : bricks < max_bricks ? (int)bricks : max_bricks);
    }
    TreeIndex view(const int32_t* mem) const {
        return TreeIndex::at(reinterpret_cast<const int2*>(mem), (uint32_t)(bricks / 2), level);
    }
};

// Launches the kernels that fill an index buffer.  `marks`: only the marked table cells get
// bricks.  With a gate nothing is launched that writes unless the gate is open: `counter` then is
// two words that hold 0, and do so again afterwards.
static int build_index(const svoxb_tree* t, const IndexLayout& l, float thresh, int softplus,
                       int32_t* mem, LogGate gate, cudaStream_t s,
                       const uint8_t* marks = nullptr, int32_t* counter = nullptr) {
    // (half as many blocks where the gate is hardly ever open: launched and gone in 4 us)
    const int sms = gate.log ? sm_count() / 2 : sm_count();
    int32_t* roots = mem + l.roots;
    if (!gate.log) {
        counter = mem + l.counter;
        if (l.cap > 0) SVOXB_CUDA(cudaMemsetAsync(counter, 0, sizeof(int32_t), s));
    }
    build_table_kernel<<<index_grid(l.cells, 256, sms), 256, 0, s>>>(
        t->child, t->data, t->K, t->M, l.level, thresh, softplus, l.cap,
        reinterpret_cast<int2*>(mem), counter, roots, marks, gate);
    if (l.cap > 0)
        fill_bricks_kernel<<<index_grid((int64_t)l.cap * kBrickCells, 256, sms), 256, 0, s>>>(
            t->child, t->data, t->K, t->M, l.level, thresh, softplus, l.cap, counter, roots,
            reinterpret_cast<int2*>(mem + l.bricks), gate);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

// What the march found where it had to leave the index.
struct Walked {
    bool ok;
    uint32_t slot;
    int depth;      // of the leaf
    float raw;      // its stored density
};

// Walks `child` from `node` at level `lvl` (root: 0) to the leaf that holds the position given
// by its coordinates floor(x * 2^24).  `ok` false: the tree is damaged there, for the caller to report.
__device__ __noinline__ Walked walk_to_leaf(const int32_t* __restrict__ child,
                                            const float* __restrict__ data, int K, int64_t M,
                                            int64_t node, int lvl, int ix, int iy, int iz) {
    for (; lvl < 24; ++lvl) {
        const int b = 23 - lvl;
        const int64_t slot = node * 8 + ((((ix >> b) & 1) << 2) | (((iy >> b) & 1) << 1) |
                                         ((iz >> b) & 1));
        const int32_t e = __ldg(child + slot);
        if (e == 0) return {true, (uint32_t)slot, lvl + 1, __ldg(data + slot * K + (K - 1))};
        node += e;
        if (node < 0 || node >= M) break;
    }
    return {false, 0u, 0, 0.f};
}

}  // namespace svoxb
