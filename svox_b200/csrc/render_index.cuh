// The render index of an octree (N = 2): what a march reads instead of walking `child` from
// the root and fetching every leaf's density from its 100- to 300-byte record.
//
// Level L of the tree is a dense TABLE of 2^L cells per side; a table cell that holds a node
// gets a BRICK, the 8x8x8 grid of the three levels below it.  Both consist of one word per
// CELL and one word per 2x2x2 GROUP of cells:
//   cell word   0x00000001 .. 0x7f800000   the cell lies in a leaf that passes the density
//                                          test; the word is its density (softplus applied)
//               kWordEmpty + d             in a leaf of depth d that fails it: a sample there
//                                          needs nothing else
//               kWordFetch + d             passes it, but the density is no positive float
//                                          (possible below a negative threshold only)
//               kWordWalk                  the tree goes deeper here: walk `child`
//               negative (table only)      kWordBrick | brick id
//   group word  bits 28-31 = k, bits 0-27 = payload: with k = the last level of the grid, the
//               payload is the node whose children are the group's cells; below that, the whole
//               group lies in a leaf k levels under the grid's root, whose slot it is
// Brick cells are stored group by group (8 cells = one 32-byte sector), because consecutive
// samples of a ray stay inside a group for two or three steps.
//
// Built per call (`data` can change between any two): one thread per table cell, then one per
// brick group, each with eight independent density loads in flight.  The bound is the 32-byte
// sector of every leaf's density (266 MB for the 8.3 M leaves of a 512^3 shell).
#pragma once

#include "query.cuh"

namespace svoxb {

// A launch that is a FALLBACK for an overflowed item log: its kernels do their work only if
// the logged forward needed more chunks than the log holds (word 0 of the log counts the
// chunks it asked for), so the host can enqueue replay and fallback without knowing which of
// the two applies.  `log` null: unconditional.
struct LogGate {
    const int32_t* log = nullptr;
    int64_t capacity = 0;
    __device__ __forceinline__ bool closed() const {
        return log != nullptr && (int64_t)__ldg(log) <= capacity;
    }
};

constexpr int kBrickLevels = 3;
constexpr int kBrickCells = 512;
constexpr int kBrickGroups = kBrickCells / 8;
constexpr int kBrickWords = kBrickCells + kBrickGroups;
constexpr int64_t kIndexMaxNodes = 1 << 25;  // slots must fit the 28 bits of a group word
constexpr int kMaxBricks = 1 << 17;
constexpr int kMaxTableLevel = 7;
constexpr int kPosBits = 23;                 // position bits below the binary point, see march

constexpr int32_t kWordInf = 0x7f800000;
constexpr int32_t kWordEmpty = kWordInf;        // + depth (1 .. 31)
constexpr int32_t kWordWalk = kWordInf + 63;
constexpr int32_t kWordFetch = kWordInf + 64;   // + depth
constexpr int32_t kWordBrick = INT32_MIN;

__device__ __forceinline__ float sigmoid_ref(float x) { return 1 / (1 + expf(-x)); }
__device__ __forceinline__ float softplus_m1(float x) { return logf(1 + expf(x - 1)); }

// The index as the march sees it: one buffer of int32 words.
struct TreeIndex {
    const int32_t* table = nullptr;   // (2^level)^3 cell words, z fastest, at the start
    uint32_t groups = 0;              // from this word on: (2^(level-1))^3 group words
    uint32_t bricks = 0;              // ... and kBrickWords per brick
    int level = 0;
};

// One density out of its record.  Without the 64-byte hint the L2 fetched 128 bytes for each of
// these scattered sectors.
__device__ __forceinline__ float ld_density(const float* a) {
    float v;
    asm("ld.global.nc.L2::64B.f32 %0, [%1];" : "=f"(v) : "l"(a));
    return v;
}

__device__ __forceinline__ int32_t leaf_word(float raw, float thresh, int softplus, int depth) {
    const float sigma = softplus ? softplus_m1(raw) : raw;
    if (!(sigma > thresh)) return kWordEmpty + depth;
    const int32_t bits = __float_as_int(sigma);
    return bits > 0 ? bits : kWordFetch + depth;
}

__global__ void __launch_bounds__(256)
build_table_kernel(const int32_t* __restrict__ child, const float* __restrict__ data, int K,
                   int64_t M, int L, float thresh, int softplus, int brick_cap,
                   int32_t* __restrict__ table, int32_t* __restrict__ groups,
                   int32_t* __restrict__ counter, int32_t* __restrict__ roots, LogGate gate) {
    if (gate.closed()) return;
    const bool fits = M < kIndexMaxNodes;
    const int S = (1 << L) - 1;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (1 << (3 * L));
         idx += gridDim.x * blockDim.x) {
        const int iz = idx & S, iy = (idx >> L) & S, ix = idx >> (2 * L);
        int64_t node = 0;
        int32_t word = kWordWalk;
        uint32_t group = 0xf0000000u;
        for (int l = 0; l < L; ++l) {
            const int b = L - 1 - l;
            const int64_t slot = node * 8 + ((((ix >> b) & 1) << 2) | (((iy >> b) & 1) << 1) |
                                             ((iz >> b) & 1));
            if (b == 0 && fits) group = ((uint32_t)l << 28) | (uint32_t)node;
            const int32_t e = __ldg(child + slot);
            if (e == 0) {
                if (b != 0 && fits) group = ((uint32_t)l << 28) | (uint32_t)slot;
                word = leaf_word(ld_density(data + slot * K + (K - 1)), thresh, softplus, l + 1);
                if (!fits && (word <= kWordInf || word >= kWordFetch)) word = kWordWalk;
                break;
            }
            node += e;
            if (node < 0 || node >= M) break;             // corrupt: reported by the march
            if (b == 0 && brick_cap > 0) {
                const int id = atomicAdd(counter, 1);
                if (id < brick_cap) {
                    roots[id] = (int32_t)node;
                    word = kWordBrick | id;
                }
            }
        }
        table[idx] = word;
        if (((ix | iy | iz) & 1) == 0)
            groups[((((ix >> 1) << (L - 1)) + (iy >> 1)) << (L - 1)) + (iz >> 1)] = (int32_t)group;
    }
}

// One thread per 2x2x2 group of a brick.
__global__ void __launch_bounds__(256)
fill_bricks_kernel(const int32_t* __restrict__ child, const float* __restrict__ data, int K,
                   int64_t M, int L, float thresh, int softplus, int cap,
                   const int32_t* __restrict__ counter, const int32_t* __restrict__ roots,
                   int32_t* __restrict__ bricks, LogGate gate) {
    if (gate.closed()) return;
    int n = *counter;
    if (n > cap) n = cap;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n * kBrickGroups;
         i += gridDim.x * blockDim.x) {
        const int g = i & (kBrickGroups - 1);
        const int gx = g >> 4, gy = (g >> 2) & 3, gz = g & 3;
        int64_t node = __ldg(roots + (i >> 6));
        int32_t w[8];
        uint32_t group = 0xf0000000u;
        int state = 0;                         // 0: on the way down, 1: words done
#pragma unroll
        for (int l = 0; l < kBrickLevels - 1; ++l) {
            if (state == 0) {
                const int b = kBrickLevels - 2 - l;
                const int64_t slot = node * 8 + ((((gx >> b) & 1) << 2) |
                                                 (((gy >> b) & 1) << 1) | ((gz >> b) & 1));
                const int32_t e = __ldg(child + slot);
                int32_t word = kWordWalk;
                if (e == 0) {
                    word = leaf_word(ld_density(data + slot * K + (K - 1)), thresh, softplus, L + 1 + l);
                    group = ((uint32_t)l << 28) | (uint32_t)slot;
                    state = 1;
                } else {
                    node += e;
                    if (node < 0 || node >= M) state = 1;      // corrupt: reported by the march
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) w[c] = word;
            }
        }
        if (state == 0) {
            group = ((uint32_t)(kBrickLevels - 1) << 28) | (uint32_t)node;
            int32_t e[8];
            float raw[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) e[c] = __ldg(child + node * 8 + c);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                raw[c] = e[c] == 0 ? ld_density(data + (node * 8 + c) * K + (K - 1)) : 0.f;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                w[c] = e[c] == 0 ? leaf_word(raw[c], thresh, softplus, L + kBrickLevels) : kWordWalk;
        }
        int32_t* __restrict__ brick = bricks + (size_t)(i >> 6) * kBrickWords;
        int4* __restrict__ out = reinterpret_cast<int4*>(brick + 8 * g);
        out[0] = make_int4(w[0], w[1], w[2], w[3]);
        out[1] = make_int4(w[4], w[5], w[6], w[7]);
        brick[kBrickCells + g] = (int32_t)group;
    }
}

// Grid of an index-building kernel over n items: enough blocks to fill the device, not one
// per 256 items (a launch that finds its gate closed should cost next to nothing).
inline unsigned index_grid(int64_t n, int block, int sms) {
    const int64_t need = (n + block - 1) / block, most = (int64_t)sms * (2048 / block) * 2;
    return (unsigned)(need < most ? (need > 0 ? need : 1) : most);
}

// Where the parts of the index lie in its buffer (int32 words, 128-byte aligned parts):
// table | groups | brick counter | brick roots | bricks.
struct IndexLayout {
    int level = 0, cap = 0;
    int64_t cells = 0;
    size_t groups = 0, counter = 0, roots = 0, bricks = 0, words = 0;

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
        l.groups = (size_t)l.cells;
        l.counter = up(l.groups + (size_t)l.cells / 8);
        l.roots = l.counter + 32;
        l.bricks = up(l.roots + (size_t)l.cap);
        l.words = l.bricks + (size_t)l.cap * kBrickWords;
        return l;
    }
    TreeIndex view(const int32_t* mem) const {
        return TreeIndex{mem, (uint32_t)groups, (uint32_t)bricks, level};
    }
};

// Launches the kernels that fill an index buffer.
static int build_index(const svoxb_tree* t, const IndexLayout& l, float thresh, int softplus,
                       int32_t* mem, LogGate gate, cudaStream_t s) {
    const int sms = sm_count();
    int32_t* counter = mem + l.counter;
    int32_t* roots = mem + l.roots;
    if (l.cap > 0) SVOXB_CUDA(cudaMemsetAsync(counter, 0, sizeof(int32_t), s));
    build_table_kernel<<<index_grid(l.cells, 256, sms), 256, 0, s>>>(
        t->child, t->data, t->K, t->M, l.level, thresh, softplus, l.cap, mem, mem + l.groups,
        counter, roots, gate);
    if (l.cap > 0)
        fill_bricks_kernel<<<index_grid((int64_t)l.cap * kBrickGroups, 256, sms), 256, 0, s>>>(
            t->child, t->data, t->K, t->M, l.level, thresh, softplus, l.cap, counter, roots,
            mem + l.bricks, gate);
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
// by its coordinates floor(x * 2^24).
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
    report(SVOXB_ERR_TREE);
    return {false, 0u, 0, 0.f};
}

}  // namespace svoxb
