// C-ABI entry points of libsvox_b200 (see include/svox_b200.h) and the
// dispatch from run-time record layouts to the templated sm_100a kernels.
// The library is this single translation unit.
#include "common.cuh"
#include "host.cuh"
#include "query.cuh"
#include "render.cuh"
#include "render_queue.cuh"
#include "render_back.cuh"
#include "render_replay.cuh"
#include "collective.cuh"
#include <initializer_list>
#include <new>

namespace svoxb {

// Queue kernels: idle lanes of a warp before it drains its queue and refills (5 measured level on
// ray batches and 2 % slower on 1080p views, 12 1 % slower on both).
constexpr int kRefillLanes = 8;
// Rays up to which the marching fallback of a replay walks the tree.  Measured (backward of an
// overflowed log, 512^3 shell, SH9): 8192 rays 0.75 ms walking, 0.54 with an index, 65536 1.40 and
// 0.92, 2^18 3.19 and 2.32, 2^20 10.3 and 8.0.  The index would pay earlier, if the log overflowed
// at every call; but its two closed launches take 8 us of every other call (3 % of a step with
// 65536 rays of an RGBA tree, 0.5 % with 2^18 of the shell).
constexpr int64_t kWalkRays = 1 << 17;
// Quarters of the leaf slots a batch has to touch for its log to be sorted.
constexpr int kSortTouches = 1;

struct RenderCall {
    const svoxb_tree* tree;
    svoxb_render_options opt;
    int64_t Q;
    // forward
    float* out = nullptr;
    // backward
    bool backward = false;
    const float* grad_out = nullptr;
    const float* fwd_out = nullptr;
    float* grad_data = nullptr;
    cudaStream_t stream = nullptr;
    // item log (logged forward / replay backward)
    int32_t* log = nullptr;
    int64_t log_capacity = 0;
    // forward with a scratch built earlier by svoxb_render_scratch_build (else per call)
    const int32_t* prepared = nullptr;
    // logged forward: buffers like `data` to clear on `clear_stream` beside the march
    float* clear[2] = {nullptr, nullptr};
    cudaStream_t clear_stream = nullptr;
    // marching backward as the fallback of a replay: does its work only if this log cannot be used
    LogGate gate{};
};

static int out_dim_of(const svoxb_tree* t, const svoxb_render_options& o) {
    // get_out_data_dim, svox/csrc/rt_kernel.cu:1009-1015
    return o.format != SVOXB_FORMAT_RGBA ? (t->K - 1) / o.basis_dim : t->K - 1;
}

// Whether the queue kernels are compiled for the records: three colour channels of basis_dim
// coefficients each and a density, or plain RGBA.
static bool queue_layout(const svoxb_tree* t, const svoxb_render_options& o) {
    const int b = o.basis_dim;
    if (o.format == SVOXB_FORMAT_RGBA) return t->K == 4;
    return t->K == 3 * b + 1 && (b == 1 || b == 4 || b == 9 || b == 16 || b == 25);
}

// Calls f with the kernels' basis size (0: RGBA) as a compile-time constant.
template <int N>
struct Basis { static constexpr int value = N; };
template <class F>
static int with_basis(const svoxb_render_options& o, F f) {
    if (o.format == SVOXB_FORMAT_RGBA) return f(Basis<0>{});
    switch (o.basis_dim) {
        case 1: return f(Basis<1>{});
        case 4: return f(Basis<4>{});
        case 9: return f(Basis<9>{});
        case 16: return f(Basis<16>{});
        case 25: return f(Basis<25>{});
    }
    return SVOXB_ERR_FORMAT;
}

static int validate_options(const svoxb_tree* t, const svoxb_render_options& o) {
    if (!(o.step_size >= 0.f)) return SVOXB_ERR_OPTION;
    if (o.format < SVOXB_FORMAT_RGBA || o.format > SVOXB_FORMAT_ASG) return SVOXB_ERR_FORMAT;
    if (o.format != SVOXB_FORMAT_RGBA) {
        const int b = o.basis_dim;
        if (o.format == SVOXB_FORMAT_SH) {
            if (b != 1 && b != 4 && b != 9 && b != 16 && b != 25) return SVOXB_ERR_FORMAT;
        } else {
            // the reference keeps the basis in an array of 25 (svox/csrc/rt_kernel.cu:253)
            if (b < 1 || b > 25) return SVOXB_ERR_FORMAT;
            if (!t->extra_data) return SVOXB_ERR_NULL;
            if (t->extra_rows < b || t->extra_cols < (o.format == SVOXB_FORMAT_SG ? 4 : 11))
                return SVOXB_ERR_SHAPE;
        }
        if (o.min_comp < 0 || o.max_comp >= b) return SVOXB_ERR_OPTION;
        if (t->K - 1 < b) return SVOXB_ERR_SHAPE;
    } else if (t->K < 2) {
        return SVOXB_ERR_SHAPE;
    }
    const int od = out_dim_of(t, o);
    if (od < 1) return SVOXB_ERR_SHAPE;
    if (o.ndc_width >= 0 && (o.ndc_width == 0 || o.ndc_height <= 0)) return SVOXB_ERR_OPTION;
    return SVOXB_OK;
}

template <class Kernel>
static int persistent_grid(Kernel kernel, int block, size_t smem, int64_t n_gran, unsigned* grid) {
    int per_sm = 0;
    const int st = blocks_per_sm(reinterpret_cast<const void*>(kernel), block, smem, &per_sm);
    if (st) return st;
    int sms = sm_count() - g_reserved_sms;     // see svoxb_reserve_sms
    if (sms < 1) sms = 1;
    int64_t g = (int64_t)sms * per_sm;
    const int64_t need = (n_gran * 32 + block - 1) / block;  // blocks that can get a granule each
    if (g > need) g = need;
    if (g < 1) g = 1;
    *grid = (unsigned)g;
    return SVOXB_OK;
}

template <int BD, bool VEC, int BLOCK, class Source>
static int launch_sh(const RenderCall& c, const Source& src, const TopTable& top, bool in_smem,
                     size_t smem) {
    const TreeArgs tr = tree_args(c.tree);
    const int64_t n_gran = (c.Q + 31) / 32;
    unsigned grid = 1;
    int st;
    if (!c.backward) {
        auto k = render_fwd_sh<BD, VEC, BLOCK, Source>;
        if ((st = persistent_grid(k, BLOCK, smem, n_gran, &grid))) return st;
        k<<<grid, BLOCK, smem, c.stream>>>(tr, src, c.opt, top, in_smem, c.out, c.Q);
    } else if (c.fwd_out != nullptr && c.opt.sigma_thresh == 0.f && c.opt.stop_thresh == 0.f) {
        auto k = render_bwd_sh<BD, VEC, BLOCK, true, Source>;
        if ((st = persistent_grid(k, BLOCK, smem, n_gran, &grid))) return st;
        k<<<grid, BLOCK, smem, c.stream>>>(tr, src, c.opt, top, in_smem, c.grad_out, c.fwd_out,
                                          c.grad_data, c.Q);
    } else {
        auto k = render_bwd_sh<BD, VEC, BLOCK, false, Source>;
        if ((st = persistent_grid(k, BLOCK, smem, n_gran, &grid))) return st;
        k<<<grid, BLOCK, smem, c.stream>>>(tr, src, c.opt, top, in_smem, c.grad_out, nullptr,
                                          c.grad_data, c.Q);
    }
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

// Log bins: a bin is a range of 2^shift leaf slots whose gradient spans
// about g_tuning.replay_bin_mb MB, at most kMaxBins of them.
static int replay_bin_shift(int64_t M, int K) {
    const int64_t per_bin = ((int64_t)g_tuning.replay_bin_mb << 20) / (K * 4);
    int shift = 2;               // a bin of the gradient is a whole number of 16-byte words
    while ((2LL << shift) <= per_bin) ++shift;
    while (((M * 8 - 1) >> shift) + 1 > kMaxBins) ++shift;
    return shift;
}
static int replay_bins(int64_t M, int K) {
    return (int)(((M * 8 - 1) >> replay_bin_shift(M, K)) + 1);
}

// Whether a logged forward sorts its items into bins: when the gradient outgrows a bin and a
// good part of it is touched (64 contributing samples per ray of a random batch, 24 per pixel,
// against the leaf slots: the averages of the 512^3 shell scene, the only one measured).  Then the
// scatter finds the gradient in L2 and clears it on the way.
// (A log of 2^26 chunks, 100 GB, or more is not sorted: no such size has been run.)
static bool sorts_log(const svoxb_tree* t, int64_t rays, bool image, int64_t capacity) {
    if (capacity / kSortedChunks >= 0xffffff || replay_bins(t->M, t->K) < 2) return false;
    return g_tuning.replay_bin_mb != kReplayBinMB ||
           rays * (image ? 24 : 64) >= kSortTouches * 8 * t->M / 4;
}

// How the queue kernels deal out `tickets` rays.  With fewer rays than fill the device's warps
// a warp takes fewer of them, so that every SM sub-partition has work: a march is a serial
// chain, and what cannot be hidden by other warps should at least run side by side.
static MarchShape march_shape(int64_t tickets, int64_t warps) {
    MarchShape m{32, 5, kRefillLanes};
    while (m.lanes > 4 && tickets <= warps * (m.lanes / 2)) m.lanes /= 2;
    // as many as two warps take, so that the blocks get alike shares (20 000 rays, SH16, 19 warps of 8
    // lanes per block: granules of 32 left some blocks with more rays than lanes, 154 us instead of
    // 135; granules of one warp: 4096 rays of a toy scene 31.5 instead of 28.8)
    while ((1 << m.granule_shift) > 2 * m.lanes) --m.granule_shift;
    if (m.lanes < 32) m.refill = m.lanes / 4;
    return m;
}

template <int BD, int MODE, int BLOCK, class Source>
static int launch_march(const RenderCall& c, const Source& src, const TreeIndex& index,
                        LogArgs log) {
    constexpr bool SORTED = BLOCK > kMarchBlock;
    constexpr size_t queues = (BLOCK / 32) * sizeof(WarpQueue<BD, MODE>);
    const int64_t tickets = Source::tickets(src, c.Q);
    const MarchShape shape = march_shape(
        tickets, (int64_t)sm_count() * (SORTED ? BLOCK / 32 : kSpreadWarps));
    auto k = render_queue_kernel<BD, MODE, BLOCK, Source>;
    unsigned grid = 1;
    const int64_t granules = (tickets + (1 << shape.granule_shift) - 1) >> shape.granule_shift;
    // One granule per block at least (persistent_grid counts granules of 32 threads).  A sorting
    // block has its SM to itself with any number of bins, so its grid is that of the most bins, and
    // is looked up once; the launch asks for no more than it needs, for the L1's sake (two bins more,
    // and the march of 2^19 rays, SH16, 62 bins, takes 2.96 ms instead of 2.26).
    int st = persistent_grid(k, BLOCK, queues + (SORTED ? kBinSmem : 0), granules * (BLOCK / 32), &grid);
    if (st) return st;
    const size_t smem = queues + (SORTED ? bin_smem(log.n_bins) : 0);
    k<<<grid, BLOCK, smem, c.stream>>>(tree_args(c.tree), src, c.opt, index, tickets, c.out, log,
                                       shape);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

template <int BD, class Source>
static int launch_back(const RenderCall& c, const Source& src, const TreeIndex& index) {
    constexpr size_t queues = (kMarchBlock / 32) * sizeof(BackQueue<BD>);
    const int64_t tickets = Source::tickets(src, c.Q);
    const MarchShape shape = march_shape(tickets, (int64_t)sm_count() * kSpreadWarps);
    auto k = render_back_kernel<BD, Source>;
    unsigned grid = 1;
    const int64_t granules = (tickets + (1 << shape.granule_shift) - 1) >> shape.granule_shift;
    const int st = persistent_grid(k, kMarchBlock, queues, granules * (kMarchBlock / 32), &grid);
    if (st) return st;
    const bool single = c.fwd_out != nullptr && c.opt.sigma_thresh == 0.f && c.opt.stop_thresh == 0.f;
    k<<<grid, kMarchBlock, queues, c.stream>>>(tree_args(c.tree), src, c.opt, index, tickets,
                                               c.grad_out, single ? c.fwd_out : nullptr, c.grad_data,
                                               c.gate, shape);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

template <int BD, class Source>
static int launch_mode(const RenderCall& c, const Source& src, const TreeIndex& index) {
    if (c.backward) return launch_back<BD>(c, src, index);
    LogArgs log;
    const bool few = Source::tickets(src, c.Q) <= (int64_t)sm_count() * kSpreadWarps * 32;
    if (c.log == nullptr)
        return few ? launch_march<BD, kModeForward, kFewBlock>(c, src, index, log)
                   : launch_march<BD, kModeForward, kMarchBlock>(c, src, index, log);
    log.log = c.log;
    log.capacity = c.log_capacity;
    log.shift = replay_bin_shift(c.tree->M, c.tree->K);
    if (!sorts_log(c.tree, c.Q, Source::kImage, c.log_capacity))
        return few ? launch_march<BD, kModeForwardLogged, kFewBlock>(c, src, index, log)
                   : launch_march<BD, kModeForwardLogged, kMarchBlock>(c, src, index, log);
    log.n_bins = replay_bins(c.tree->M, c.tree->K);
    const int st = launch_march<BD, kModeForwardLogged, sorted_march_block<BD>()>(c, src, index, log);
    if (st) return st;
    int32_t* cursor = c.log + log_words(c.log_capacity) - kMaxBins;
    SVOXB_CUDA(cudaMemsetAsync(cursor, 0, kMaxBins * sizeof(int32_t), c.stream));
    order_groups_kernel<<<index_grid(c.log_capacity / kSortedChunks, kOrderTile, sm_count()), 256,
                          0, c.stream>>>(c.log, c.log_capacity, cursor);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

// Replay backward (render_replay.cuh) in one or several parts (bin ranges).
struct ReplayJob {
    int32_t* log = nullptr;
    int64_t capacity = 0;
    int64_t chunks = 0;          // at most this many are in the log
    svoxb_render_options opt{};
    TreeArgs tree{};
    ScatterOut to{};
    int64_t n_slots = 0;
    int n_parts = 1, shift = 0, n_bins = 1;
};

static int replay_job(const RenderCall& c, int64_t chunks, int n_parts, ReplayJob* job) {
    if (n_parts < 1 || n_parts > kMaxParts) return SVOXB_ERR_OPTION;
    job->log = c.log;
    job->capacity = c.log_capacity;
    job->chunks = chunks > c.log_capacity ? c.log_capacity : chunks;
    job->opt = c.opt;
    job->tree = tree_args(c.tree);
    job->to = ScatterOut{c.grad_data, nullptr, c.grad_out, c.fwd_out, 0};
    job->n_slots = c.tree->M * 8;
    job->n_parts = n_parts;
    job->shift = replay_bin_shift(c.tree->M, c.tree->K);
    job->n_bins = replay_bins(c.tree->M, c.tree->K);
    return SVOXB_OK;
}

// Scatter of one part.  With `reserve_sms` > 0 that many SMs are left without a block (for a
// collective that runs beside the scatter); one 1024-thread block per SM then, so that the SMs
// left out are really empty.
template <int BD, int BLOCK, bool HESS, bool LOBES>
static int replay_scatter_block(const ReplayJob& job, int part, int reserve_sms,
                                cudaStream_t stream) {
    constexpr int K = RecordLength<BD>::K;
    const size_t smem = (size_t)(BLOCK / 32) * sizeof(ScatterSmem<K>);
    auto k = replay_scatter_kernel<BD, BLOCK, HESS, LOBES>;
    // blocks for the clearing too, which few packets may come with
    const int64_t clears = job.to.zero_slots * K / kZeroFloats * (BLOCK / 32);
    unsigned grid = 1;
    int st = persistent_grid(k, BLOCK, smem, job.chunks > clears ? job.chunks : clears, &grid);
    if (st) return st;
    // Two outputs to clear: with more than two blocks per SM the units of adding come round to a bin
    // before it is cleared, and wait.  Measured (`se_grad`, 512^3 shell, 10.5 M records, ms with 2 / 3 / as
    // many blocks as fit; 1 block is slower everywhere but for 45 000 rays of SH16, 1.86 against 1.91):
    //            45 000 rays         100 000             300 000             2^20
    //     RGBA   0.57 / 0.59 / 0.59  0.75 / 0.76 / 0.76  1.60 / 1.59 / 1.60  4.78 / 4.73 / 4.75
    //     SH4    0.84 / 0.90 / 0.92  1.11 / 1.12 / 1.16  2.20 / 2.21 / 2.21  6.53 / 6.39 / 6.40
    //     SH9    1.20 / 1.43 / 1.43  1.58 / 1.70 / 1.70  2.98 / 2.98 / 2.98  7.76 / 7.84 / 7.86
    //     SH16   1.91 / 1.91 / 1.91  2.50 / 2.50 / 2.50  4.40 / 4.40 / 4.40
    // So two, or three where many samples (64 a ray) come to a short record.  One output: the 2^20-ray
    // step with 1 / 2 / 3 / 4 / 6 blocks 3.05, 2.05, 1.90, 1.90, 2.34.
    if (HESS && job.to.grad != nullptr && job.to.zero_slots > 0) {
        const bool many = K <= 13 && 32 * job.chunks > 4 * job.to.zero_slots;
        const int64_t most = (many ? 3LL : 2LL) * (sm_count() - g_reserved_sms);
        if ((int64_t)grid > most && most > 0) grid = (unsigned)most;
    }
    if (reserve_sms > 0) {
        const int sms = sm_count();
        const int64_t per_sm = ((int64_t)grid + sms - 1) / sms;
        const int64_t most = ((int64_t)sms - reserve_sms) * per_sm;
        if ((int64_t)grid > most) grid = (unsigned)(most > 1 ? most : 1);
    }
    k<<<grid, BLOCK, smem, stream>>>(job.tree, job.opt, job.log, job.capacity, job.to, part,
                                    job.n_parts);
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? set_cuda_error(e) : SVOXB_OK;
}

template <int BD, bool LOBES>
static int replay_scatter_bd(const ReplayJob& job, int part, int reserve_sms,
                             cudaStream_t stream) {
    if (job.to.hess != nullptr)
        return replay_scatter_block<BD, kScatterBlock, true, LOBES>(job, part, 0, stream);
    if constexpr (BD <= 9 && !LOBES) {
        if (reserve_sms > 0)
            return replay_scatter_block<BD, 1024, false, LOBES>(job, part, reserve_sms, stream);
    }
    return replay_scatter_block<BD, kScatterBlock, false, LOBES>(job, part, reserve_sms, stream);
}

static int replay_scatter(const ReplayJob& job, int part, int reserve_sms, cudaStream_t stream) {
    if (part < 0 || part >= job.n_parts) return SVOXB_ERR_OPTION;
    if (job.chunks < 1) return SVOXB_OK;
    return with_basis(job.opt, [&](auto basis) {
        constexpr int BD = decltype(basis)::value;
        if constexpr (BD > 0) {
            if (job.opt.format != SVOXB_FORMAT_SH)
                return replay_scatter_bd<BD, true>(job, part, reserve_sms, stream);
        }
        return replay_scatter_bd<BD, false>(job, part, reserve_sms, stream);
    });
}

// The index of one call (render_index.cuh): a pool allocation, freed on the stream.
struct QueueScratch {
    int32_t* mem = nullptr;
    cudaStream_t stream = nullptr;

    static IndexLayout layout(const svoxb_tree* t) {
        return IndexLayout::of(t->M, g_tuning.render_bricks ? kMaxBricks : 0);
    }
    // A batch of few rays touches few of a large tree's bricks: those it passes are marked first
    // (10 us) and only they are filled (1.3 M nodes: 115 us for all).  (512 rays of the
    // 512^3 shell scene: 320 us in all before, 230 after.)
    static constexpr int64_t kMarkRays = 1024, kMarkNodes = 1 << 18;

    template <class Source>
    int build(const RenderCall& c, const Source& src, const IndexLayout& l) {
        const svoxb_tree* t = c.tree;
        stream = c.stream;
        int st = keep_pool_cached();
        if (st) return st;
        const bool mark = c.Q <= kMarkRays && t->M >= kMarkNodes && l.cap > 0;
        SVOXB_CUDA(cudaMallocAsync((void**)&mem, l.words * sizeof(int32_t) + (mark ? l.cells : 0),
                                   stream));
        uint8_t* marks = mark ? reinterpret_cast<uint8_t*>(mem + l.words) : nullptr;
        if (mark) {
            SVOXB_CUDA(cudaMemsetAsync(marks, 0, (size_t)l.cells, stream));
            const int64_t tickets = Source::tickets(src, c.Q);
            mark_cells_kernel<<<(unsigned)((tickets + 3) / 4), 128, 0, stream>>>(
                tree_args(t), src, c.opt, tickets, l.level, marks);
        }
        return build_index(t, l, c.backward ? 0.f : c.opt.sigma_thresh, c.opt.density_softplus,
                           mem, LogGate{}, stream, marks);
    }
    ~QueueScratch() { if (mem) cudaFreeAsync(mem, stream); }
};

// Clears the buffers of a logged forward once the index is built, behind the launch of the march,
// which leaves most of the memory bandwidth and many places on the SMs unused.  (Started before
// the index the fill put its blocks in front of it and delayed the march by all of its time.)
struct ClearBeside {
    const RenderCall& c;
    cudaEvent_t ready = nullptr;

    int index_built() {
        if (!c.clear[0]) return SVOXB_OK;
        SVOXB_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
        SVOXB_CUDA(cudaEventRecord(ready, c.stream));
        return SVOXB_OK;
    }
    int march_launched() {
        if (!c.clear[0]) return SVOXB_OK;
        SVOXB_CUDA(cudaStreamWaitEvent(c.clear_stream, ready, 0));
        const size_t n = (size_t)c.tree->M * 8 * (size_t)c.tree->K;
        for (float* to : c.clear)
            if (to) SVOXB_CUDA(cudaMemsetAsync(to, 0, n * sizeof(float), c.clear_stream));
        return SVOXB_OK;
    }
    ~ClearBeside() { if (ready) cudaEventDestroy(ready); }
};

// The index for the marching fallback of a replay, which does its work only if the log turned out
// to be of no use: built, in that case, in the log's own memory, with as many bricks as fit.  Up to
// kWalkRays rays, or without room for the table, the march walks the tree instead (`mem` stays
// null).
static int fallback_index(const RenderCall& c, IndexLayout* layout, const int32_t** mem) {
    const int64_t capacity = c.gate.capacity, at = log_packets_at(capacity);
    const int64_t room = log_words(capacity) - at;
    *mem = nullptr;
    if (c.Q <= kWalkRays) return SVOXB_OK;
    *layout = IndexLayout::within(c.tree->M, g_tuning.render_bricks ? kMaxBricks : 0, room);
    if ((int64_t)layout->words > room) return SVOXB_OK;
    int32_t* log = const_cast<int32_t*>(c.gate.log);
    const int st = build_index(c.tree, *layout, 0.f, c.opt.density_softplus, log + at, c.gate,
                               c.stream, nullptr, log + kLogBricks);
    if (st == SVOXB_OK) *mem = log + at;
    return st;
}

template <class Source>
static int launch_queue(const RenderCall& c, const Source& src) {
    IndexLayout layout = QueueScratch::layout(c.tree);
    QueueScratch scratch;
    const int32_t* mem = c.prepared;
    int st = SVOXB_OK;
    if (c.gate.log != nullptr) {
        if ((st = fallback_index(c, &layout, &mem))) return st;
    } else if (mem == nullptr || c.backward) {
        if ((st = scratch.build(c, src, layout))) return st;
        mem = scratch.mem;
    }
    TreeIndex index = layout.view(mem);
    if (mem == nullptr) index = TreeIndex::at(nullptr, 0, 1);
    ClearBeside clear{c};
    if ((st = clear.index_built())) return st;
    st = with_basis(c.opt, [&](auto basis) {
        constexpr int BD = decltype(basis)::value;
        if constexpr (BD > 0) {
            if (c.opt.format != SVOXB_FORMAT_SH)
                return launch_mode<BD>(c, WithLobes<Source>{src}, index);
        }
        return launch_mode<BD>(c, src, index);
    });
    return st ? st : clear.march_launched();
}

template <int BLOCK, class Source>
static int launch_generic(const RenderCall& c, const Source& src, const TopTable& top,
                          bool in_smem, size_t smem) {
    const TreeArgs tr = tree_args(c.tree);
    const int64_t n_gran = (c.Q + 31) / 32;
    const int od = out_dim_of(c.tree, c.opt);
    if (od > kMaxGenericOut) return SVOXB_ERR_FORMAT;
    unsigned grid = 1;
    int st;
    if (!c.backward) {
        auto k = render_fwd_generic<BLOCK, Source>;
        if ((st = persistent_grid(k, BLOCK, smem, n_gran, &grid))) return st;
        k<<<grid, BLOCK, smem, c.stream>>>(tr, src, c.opt, top, in_smem, c.out, c.Q, od);
    } else {
        auto k = render_bwd_generic<BLOCK, Source>;
        if ((st = persistent_grid(k, BLOCK, smem, n_gran, &grid))) return st;
        k<<<grid, BLOCK, smem, c.stream>>>(tr, src, c.opt, top, in_smem, c.grad_out, c.grad_data,
                                          c.Q, od);
    }
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

template <int BLOCK, class Source>
static int dispatch_layout(const RenderCall& c, const Source& src, const TopTable& top,
                           bool in_smem, size_t smem) {
    const svoxb_tree* t = c.tree;
    const bool sh3 = queue_layout(t, c.opt) && c.opt.format == SVOXB_FORMAT_SH;
    if (!sh3) return launch_generic<BLOCK>(c, src, top, in_smem, smem);
    const bool aligned = ((uintptr_t)t->data % 16 == 0) &&
                         (!c.backward || (uintptr_t)c.grad_data % 16 == 0);
    const bool vec = aligned && (t->K % 4 == 0);
    switch (c.opt.basis_dim) {
        case 1:
            return vec ? launch_sh<1, true, BLOCK>(c, src, top, in_smem, smem)
                       : launch_sh<1, false, BLOCK>(c, src, top, in_smem, smem);
        case 4: return launch_sh<4, false, BLOCK>(c, src, top, in_smem, smem);
        case 9:
            return vec ? launch_sh<9, true, BLOCK>(c, src, top, in_smem, smem)
                       : launch_sh<9, false, BLOCK>(c, src, top, in_smem, smem);
        case 16: return launch_sh<16, false, BLOCK>(c, src, top, in_smem, smem);
        case 25:
            return vec ? launch_sh<25, true, BLOCK>(c, src, top, in_smem, smem)
                       : launch_sh<25, false, BLOCK>(c, src, top, in_smem, smem);
    }
    return SVOXB_ERR_FORMAT;
}

template <class Source>
static int render_dispatch(const RenderCall& c, const Source& src) {
    int st = validate_tree(c.tree);
    if (st) return st;
    if ((st = validate_options(c.tree, c.opt))) return st;
    if (c.Q < 0) return SVOXB_ERR_SHAPE;
    if (c.backward) {
        if (!c.grad_data) return SVOXB_ERR_NULL;
    }
    if (c.Q == 0) return SVOXB_OK;
    if (c.backward ? !c.grad_out : !c.out) return SVOXB_ERR_NULL;

    // Default path: the queue kernels, for octrees with records they are compiled for, in
    // buffers that allow the record's 16-byte words.
    {
        const svoxb_tree* t = c.tree;
        const bool aligned = ((uintptr_t)t->data % 16 == 0) &&
                             (!c.backward || (uintptr_t)c.grad_data % 16 == 0);
        if (queue_layout(t, c.opt) && t->N == 2 && (aligned || t->K % 4 != 0) &&
            t->M < (1LL << 28))
            return launch_queue(c, src);
    }

    TopScratch scratch;
    if ((st = scratch.build(c.tree, 5, c.stream))) return st;
    const TopTable top{scratch.cells, scratch.level};
    // The table is staged in shared memory up to level 5 (128 KB).
    const bool in_smem = scratch.level > 0 && scratch.level <= 5;
    const size_t smem = in_smem ? ((size_t)4 << (3 * scratch.level)) : 0;
    if (smem > 64 * 1024) return dispatch_layout<1024>(c, src, top, in_smem, smem);
    return dispatch_layout<256>(c, src, top, in_smem, smem);
}

static int zero_grad(const svoxb_tree* t, float* grad, int K, cudaStream_t s) {
    const size_t n = (size_t)t->M * t->N * t->N * t->N * (size_t)K;
    SVOXB_CUDA(cudaMemsetAsync(grad, 0, n * sizeof(float), s));
    return SVOXB_OK;
}

}  // namespace svoxb

using namespace svoxb;

extern "C" {

int svoxb_query_vertical(const svoxb_tree* tree, const float* indices, int64_t Q,
                         float* values_out, int64_t* node_ids_out, void* stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if (Q < 0) return SVOXB_ERR_SHAPE;
    return launch_query(tree, indices, Q, values_out, node_ids_out, nullptr, nullptr, 0,
                        (cudaStream_t)stream);
}

int svoxb_query_vertical_backward(const svoxb_tree* tree, const float* indices, int64_t Q,
                                  const float* grad_output, int32_t Kg, float* grad_data_out,
                                  int zero_first, void* stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if (Q < 0 || Kg < 1) return SVOXB_ERR_SHAPE;
    if (!grad_data_out || (Q > 0 && !grad_output)) return SVOXB_ERR_NULL;
    if (Q > 0 && !indices) return SVOXB_ERR_NULL;
    return launch_query_backward(tree, indices, Q, grad_output, Kg, grad_data_out, zero_first != 0,
                                 (cudaStream_t)stream);
}

int svoxb_query_scatter(const svoxb_tree* tree, const int64_t* node_ids, int64_t Q,
                        const float* grad_output, int32_t Kg, float* grad_data_out, int zero_first,
                        void* stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if (Q < 0 || Kg < 1) return SVOXB_ERR_SHAPE;
    if (!grad_data_out || (Q > 0 && (!grad_output || !node_ids))) return SVOXB_ERR_NULL;
    return launch_scatter(tree, node_ids, Q, grad_output, Kg, grad_data_out, zero_first != 0,
                          (cudaStream_t)stream);
}

int svoxb_assign_vertical(const svoxb_tree* tree, const float* indices, int64_t Q,
                          const float* values, int32_t Kv, float* data_out, void* stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if (Q < 0 || Kv < 1 || Kv > tree->K) return SVOXB_ERR_SHAPE;
    if (!data_out || (Q > 0 && !values)) return SVOXB_ERR_NULL;
    return launch_query(tree, indices, Q, nullptr, nullptr, values, data_out, Kv,
                        (cudaStream_t)stream);
}

int svoxb_calc_corners(const svoxb_tree* tree, const int32_t* parent_depth,
                       const int64_t* indexer, int64_t Q, float* out, void* stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if (Q < 0) return SVOXB_ERR_SHAPE;
    if (Q == 0) return SVOXB_OK;
    if (!parent_depth || !indexer || !out) return SVOXB_ERR_NULL;
    if ((Q + 255) / 256 > 0x7fffffffLL) return SVOXB_ERR_TOO_LARGE;
    calc_corners_kernel<<<(unsigned)((Q + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        parent_depth, tree->M, tree->N, indexer, Q, out);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

int svoxb_volume_render(const svoxb_tree* tree, const svoxb_rays* rays,
                        const svoxb_render_options* opt, float* out, void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    RenderCall c{tree, *opt, rays->Q};
    c.out = out;
    c.stream = (cudaStream_t)stream;
    return render_dispatch(c, RayBatch{rays->origins, rays->dirs, rays->vdirs});
}

int svoxb_volume_render_image(const svoxb_tree* tree, const svoxb_camera* cam,
                              const svoxb_render_options* opt, float* out, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    RenderCall c{tree, *opt, (int64_t)cam->width * cam->height};
    c.out = out;
    c.stream = (cudaStream_t)stream;
    return render_dispatch(c, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height});
}

// Whether the queue kernels take this tree and these options (the prepared scratch is theirs).
static int queue_eligible(const svoxb_tree* t, const svoxb_render_options* o) {
    int st = validate_tree(t);
    if (st) return st;
    if ((st = validate_options(t, *o))) return st;
    if (!queue_layout(t, *o) || t->N != 2)
        return SVOXB_ERR_FORMAT;
    if (t->K % 4 == 0 && (uintptr_t)t->data % 16 != 0) return SVOXB_ERR_FORMAT;
    if (t->M >= (1LL << 28)) return SVOXB_ERR_TOO_LARGE;
    return SVOXB_OK;
}

int64_t svoxb_render_scratch_words(const svoxb_tree* tree) {
    if (!tree || tree->M < 1 || tree->N != 2) return 0;
    return (int64_t)QueueScratch::layout(tree).words;
}

int svoxb_render_scratch_build(const svoxb_tree* tree, const svoxb_render_options* opt,
                               int32_t* scratch, void* stream) {
    if (!tree || !opt || !scratch) return SVOXB_ERR_NULL;
    int st = queue_eligible(tree, opt);
    if (st) return st;
    return build_index(tree, QueueScratch::layout(tree), opt->sigma_thresh,
                       opt->density_softplus, scratch, LogGate{}, (cudaStream_t)stream);
}

int svoxb_volume_render_prepared(const svoxb_tree* tree, const svoxb_rays* rays,
                                 const svoxb_render_options* opt, const int32_t* scratch,
                                 float* out, void* stream) {
    if (!tree || !rays || !opt || !scratch) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    int st = queue_eligible(tree, opt);
    if (st) return st;
    RenderCall c{tree, *opt, rays->Q};
    c.out = out;
    c.stream = (cudaStream_t)stream;
    c.prepared = scratch;
    return render_dispatch(c, RayBatch{rays->origins, rays->dirs, rays->vdirs});
}

int svoxb_volume_render_image_prepared(const svoxb_tree* tree, const svoxb_camera* cam,
                                       const svoxb_render_options* opt, const int32_t* scratch,
                                       float* out, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w || !scratch) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    int st = queue_eligible(tree, opt);
    if (st) return st;
    RenderCall c{tree, *opt, (int64_t)cam->width * cam->height};
    c.out = out;
    c.stream = (cudaStream_t)stream;
    c.prepared = scratch;
    return render_dispatch(c, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height});
}

int svoxb_volume_render_backward(const svoxb_tree* tree, const svoxb_rays* rays,
                                 const svoxb_render_options* opt, const float* grad_output,
                                 const float* fwd_out, float* grad_data_out, int zero_first,
                                 void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    int st = validate_tree(tree);
    if (st) return st;
    if (!grad_data_out) return SVOXB_ERR_NULL;
    if (zero_first && (st = zero_grad(tree, grad_data_out, tree->K, (cudaStream_t)stream)))
        return st;
    RenderCall c{tree, *opt, rays->Q};
    c.backward = true;
    c.grad_out = grad_output;
    c.fwd_out = fwd_out;
    c.grad_data = grad_data_out;
    c.stream = (cudaStream_t)stream;
    return render_dispatch(c, RayBatch{rays->origins, rays->dirs, rays->vdirs});
}

int svoxb_volume_render_image_backward(const svoxb_tree* tree, const svoxb_camera* cam,
                                       const svoxb_render_options* opt,
                                       const float* grad_output, const float* fwd_out,
                                       float* grad_data_out, int zero_first, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    int st = validate_tree(tree);
    if (st) return st;
    if (!grad_data_out) return SVOXB_ERR_NULL;
    if (zero_first && (st = zero_grad(tree, grad_data_out, tree->K, (cudaStream_t)stream)))
        return st;
    RenderCall c{tree, *opt, (int64_t)cam->width * cam->height};
    c.backward = true;
    c.grad_out = grad_output;
    c.fwd_out = fwd_out;
    c.grad_data = grad_data_out;
    c.stream = (cudaStream_t)stream;
    return render_dispatch(c, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height});
}

}  // extern "C"

// Whether a call can take the logged forward / replay backward pair.
static int log_eligible(const svoxb_tree* t, const svoxb_render_options* o, const float* grad) {
    if (!queue_layout(t, *o) || t->N != 2)
        return SVOXB_ERR_FORMAT;
    if (o->sigma_thresh != 0.f || o->stop_thresh != 0.f) return SVOXB_ERR_OPTION;
    if (t->M >= (1LL << 28)) return SVOXB_ERR_TOO_LARGE;
    if (t->K % 4 == 0 && ((uintptr_t)t->data % 16 != 0 || (uintptr_t)grad % 16 != 0))
        return SVOXB_ERR_FORMAT;
    return SVOXB_OK;
}

template <class Source>
static int logged_forward(const svoxb_tree* tree, const Source& src, int64_t Q,
                          const svoxb_render_options* opt, float* out, int32_t* log,
                          int64_t capacity_chunks, void* stream, float* clear0 = nullptr,
                          float* clear1 = nullptr, void* clear_stream = nullptr) {
    int st = validate_tree(tree);
    if (st) return st;
    if ((st = validate_options(tree, *opt))) return st;
    if ((st = log_eligible(tree, opt, nullptr))) return st;
    if (!log || capacity_chunks < 1 || Q < 0) return SVOXB_ERR_SHAPE;
    if (Q > 0 && !out) return SVOXB_ERR_NULL;
    SVOXB_CUDA(cudaMemsetAsync(log, 0, kLogCounts * sizeof(int32_t), (cudaStream_t)stream));
    if (Q == 0) return SVOXB_OK;
    RenderCall c{tree, *opt, Q};
    c.out = out;
    c.stream = (cudaStream_t)stream;
    c.log = log;
    c.log_capacity = capacity_chunks;
    c.clear[0] = clear0;
    c.clear[1] = clear1;
    c.clear_stream = (cudaStream_t)clear_stream;
    return launch_queue(c, src);
}

// Gradient (`grad_data_out`) and / or Gauss-Newton diagonal (`hess_out`) from the log.
template <class Source>
static int replay_backward(const svoxb_tree* tree, const Source& src, int64_t Q,
                           const svoxb_render_options* opt, const float* grad_output,
                           const float* fwd_out, int32_t* log, int64_t capacity_chunks,
                           int64_t chunks_used, float* grad_data_out, float* hess_out,
                           int zero_first, void* stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if ((st = validate_options(tree, *opt))) return st;
    if ((!grad_data_out && !hess_out) || !log) return SVOXB_ERR_NULL;
    // a sorted log's scatter clears its outputs itself
    bool clears = zero_first && Q > 0 && sorts_log(tree, Q, Source::kImage, capacity_chunks);
    for (float* out : {grad_data_out, hess_out}) clears = clears && (uintptr_t)out % 16 == 0;
    for (float* out : {grad_data_out, hess_out}) {
        if (!out) continue;
        if ((st = log_eligible(tree, opt, out))) return st;
        if (zero_first && !clears &&
            (st = zero_grad(tree, out, tree->K, (cudaStream_t)stream)))
            return st;
    }
    if (Q == 0) return SVOXB_OK;
    if ((grad_data_out && !grad_output) || !fwd_out) return SVOXB_ERR_NULL;
    RenderCall c{tree, *opt, Q};
    c.backward = true;
    c.grad_out = grad_output;
    c.fwd_out = fwd_out;
    c.grad_data = grad_data_out;
    c.stream = (cudaStream_t)stream;
    c.log = log;
    c.log_capacity = capacity_chunks;
    // chunks_used > 0: the caller has read the count (svoxb_item_log_used) and vouches that
    // the log did not overflow.  Otherwise the count stays on the device: the kernel reads it
    // itself, and a march enqueued behind it does its work only if the log overflowed.
    const bool known = chunks_used > 0 && chunks_used <= capacity_chunks;
    if (hess_out && !grad_data_out && !known) return SVOXB_ERR_OPTION;
    ReplayJob job;
    if ((st = replay_job(c, known ? chunks_used : capacity_chunks, 1, &job))) return st;
    job.to.hess = hess_out;
    if (clears) job.to.zero_slots = job.n_slots;
    if ((st = replay_scatter(job, 0, 0, c.stream)) || known) return st;
    c.log = nullptr;
    c.gate = LogGate{log, capacity_chunks};
    if (!hess_out) return render_dispatch(c, src);
    auto k = render_se_grad_generic<256, Source>;
    unsigned grid = 1;
    if ((st = persistent_grid(k, 256, 0, (Q + 31) / 32, &grid))) return st;
    k<<<grid, 256, 0, c.stream>>>(tree_args(tree), src, *opt, TopTable{nullptr, 0}, false, fwd_out,
                                  nullptr, grad_output, grad_data_out, hess_out, Q, 3, c.gate);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

extern "C" {

int svoxb_log_is_sorted(const svoxb_tree* tree, int64_t n_rays, int image,
                        int64_t capacity_chunks) {
    if (!tree || tree->M < 1 || tree->K < 1) return 0;
    return sorts_log(tree, n_rays, image != 0, capacity_chunks) ? 1 : 0;
}

int64_t svoxb_item_log_words(int64_t capacity_chunks) {
    return log_words(capacity_chunks);
}

int svoxb_volume_render_logged(const svoxb_tree* tree, const svoxb_rays* rays,
                               const svoxb_render_options* opt, float* out, int32_t* log,
                               int64_t capacity_chunks, void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    return logged_forward(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q, opt,
                          out, log, capacity_chunks, stream);
}

int svoxb_volume_render_image_logged(const svoxb_tree* tree, const svoxb_camera* cam,
                                     const svoxb_render_options* opt, float* out, int32_t* log,
                                     int64_t capacity_chunks, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    return logged_forward(tree, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                          (int64_t)cam->width * cam->height, opt, out, log, capacity_chunks,
                          stream);
}

int svoxb_volume_render_logged_clear(const svoxb_tree* tree, const svoxb_rays* rays,
                                     const svoxb_render_options* opt, float* out, int32_t* log,
                                     int64_t capacity_chunks, void* stream, float* clear0,
                                     float* clear1, void* clear_stream) {
    if (!tree || !rays || !opt || !clear0) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    if (rays->Q <= 0) return SVOXB_ERR_SHAPE;
    return logged_forward(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q, opt,
                          out, log, capacity_chunks, stream, clear0, clear1, clear_stream);
}

int svoxb_volume_render_image_logged_clear(const svoxb_tree* tree, const svoxb_camera* cam,
                                           const svoxb_render_options* opt, float* out,
                                           int32_t* log, int64_t capacity_chunks, void* stream,
                                           float* clear0, float* clear1, void* clear_stream) {
    if (!tree || !cam || !opt || !cam->c2w || !clear0) return SVOXB_ERR_NULL;
    if (cam->width <= 0 || cam->height <= 0) return SVOXB_ERR_SHAPE;
    return logged_forward(tree, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                          (int64_t)cam->width * cam->height, opt, out, log, capacity_chunks,
                          stream, clear0, clear1, clear_stream);
}

int svoxb_volume_render_backward_replay(const svoxb_tree* tree, const svoxb_rays* rays,
                                        const svoxb_render_options* opt,
                                        const float* grad_output, const float* fwd_out,
                                        int32_t* log, int64_t capacity_chunks,
                                        int64_t chunks_used, float* grad_data_out,
                                        int zero_first, void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    return replay_backward(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q, opt,
                           grad_output, fwd_out, log, capacity_chunks, chunks_used, grad_data_out,
                           nullptr, zero_first, stream);
}

int svoxb_volume_render_image_backward_replay(const svoxb_tree* tree, const svoxb_camera* cam,
                                              const svoxb_render_options* opt,
                                              const float* grad_output, const float* fwd_out,
                                              int32_t* log, int64_t capacity_chunks,
                                              int64_t chunks_used, float* grad_data_out,
                                              int zero_first, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    return replay_backward(tree, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                           (int64_t)cam->width * cam->height, opt, grad_output, fwd_out, log,
                           capacity_chunks, chunks_used, grad_data_out, nullptr, zero_first,
                           stream);
}

/* Gauss-Newton diagonal of the squared error from the item log (the third result of the
 * reference's se_grad, svox/csrc/rt_kernel.cu:479-715, 1111-1173). */
int svoxb_volume_render_hessdiag_replay(const svoxb_tree* tree, const svoxb_rays* rays,
                                        const svoxb_render_options* opt, const float* fwd_out,
                                        int32_t* log, int64_t capacity_chunks,
                                        int64_t chunks_used, float* hessdiag_out,
                                        int zero_first, void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    return replay_backward(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q, opt,
                           nullptr, fwd_out, log, capacity_chunks, chunks_used, nullptr,
                           hessdiag_out, zero_first, stream);
}

int svoxb_volume_render_image_hessdiag_replay(const svoxb_tree* tree, const svoxb_camera* cam,
                                              const svoxb_render_options* opt,
                                              const float* fwd_out, int32_t* log,
                                              int64_t capacity_chunks, int64_t chunks_used,
                                              float* hessdiag_out, int zero_first,
                                              void* stream) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    return replay_backward(tree, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                           (int64_t)cam->width * cam->height, opt, nullptr, fwd_out, log,
                           capacity_chunks, chunks_used, nullptr, hessdiag_out, zero_first,
                           stream);
}

/* Both at once: the packets are read once. */
int svoxb_se_grad_replay(const svoxb_tree* tree, const svoxb_rays* rays,
                         const svoxb_render_options* opt, const float* residual,
                         const float* fwd_out, int32_t* log, int64_t capacity_chunks,
                         int64_t chunks_used, float* grad_data_out, float* hessdiag_out,
                         int zero_first, void* stream) {
    if (!tree || !rays || !opt || !grad_data_out || !hessdiag_out) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    return replay_backward(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q, opt,
                           residual, fwd_out, log, capacity_chunks, chunks_used, grad_data_out,
                           hessdiag_out, zero_first, stream);
}

int svoxb_se_grad_image_replay(const svoxb_tree* tree, const svoxb_camera* cam,
                               const svoxb_render_options* opt, const float* residual,
                               const float* fwd_out, int32_t* log, int64_t capacity_chunks,
                               int64_t chunks_used, float* grad_data_out, float* hessdiag_out,
                               int zero_first, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w || !grad_data_out || !hessdiag_out)
        return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    return replay_backward(tree, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                           (int64_t)cam->width * cam->height, opt, residual, fwd_out, log,
                           capacity_chunks, chunks_used, grad_data_out, hessdiag_out, zero_first,
                           stream);
}

}  // extern "C"

// se_grad by marching (any record layout the generic kernels take): gradient and
// Gauss-Newton diagonal of the squared error from the forward's output.
template <class Source>
static int se_grad_march(const svoxb_tree* tree, const Source& src, int64_t Q,
                         const svoxb_render_options* opt, const float* fwd_out,
                         const float* color_ref, float* grad, float* hess, int zero_first,
                         cudaStream_t stream) {
    int st = validate_tree(tree);
    if (st) return st;
    if ((st = validate_options(tree, *opt))) return st;
    if (Q < 0) return SVOXB_ERR_SHAPE;
    if (!grad || !hess || (Q > 0 && (!fwd_out || !color_ref))) return SVOXB_ERR_NULL;
    const int od = out_dim_of(tree, *opt);
    if (od > kMaxSeGradOut) return SVOXB_ERR_FORMAT;
    if (zero_first) {
        if ((st = zero_grad(tree, grad, tree->K, stream))) return st;
        if ((st = zero_grad(tree, hess, tree->K, stream))) return st;
    }
    if (Q == 0) return SVOXB_OK;
    TopScratch scratch;
    if ((st = scratch.build(tree, 5, stream))) return st;
    const TopTable top{scratch.cells, scratch.level};
    const bool in_smem = scratch.level > 0 && scratch.level <= 5;
    const size_t smem = in_smem ? ((size_t)4 << (3 * scratch.level)) : 0;
    const TreeArgs tr = tree_args(tree);
    const int64_t n_gran = (Q + 31) / 32;
    unsigned grid = 1;
    auto run = [&](auto k, int block) {
        int s2 = persistent_grid(k, block, smem, n_gran, &grid);
        if (s2) return s2;
        k<<<grid, block, smem, stream>>>(tr, src, *opt, top, in_smem, fwd_out, color_ref, nullptr,
                                        grad, hess, Q, od, LogGate{});
        const cudaError_t e = cudaGetLastError();
        return e != cudaSuccess ? set_cuda_error(e) : (int)SVOXB_OK;
    };
    return smem > 64 * 1024 ? run(render_se_grad_generic<1024, Source>, 1024)
                            : run(render_se_grad_generic<256, Source>, 256);
}

extern "C" {

int svoxb_se_grad_march(const svoxb_tree* tree, const svoxb_rays* rays,
                        const svoxb_render_options* opt, const float* fwd_out,
                        const float* color_ref, float* grad_data_out, float* hessdiag_out,
                        int zero_first, void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    return se_grad_march(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q, opt,
                         fwd_out, color_ref, grad_data_out, hessdiag_out, zero_first,
                         (cudaStream_t)stream);
}

int svoxb_se_grad_image_march(const svoxb_tree* tree, const svoxb_camera* cam,
                              const svoxb_render_options* opt, const float* fwd_out,
                              const float* color_ref, float* grad_data_out, float* hessdiag_out,
                              int zero_first, void* stream) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    return se_grad_march(tree, PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                         (int64_t)cam->width * cam->height, opt, fwd_out, color_ref,
                         grad_data_out, hessdiag_out, zero_first, (cudaStream_t)stream);
}

}  // extern "C"

template <class Source>
static int replay_begin_checked(const svoxb_tree* tree, const Source& src, int64_t Q,
                                const svoxb_render_options* opt, const float* grad_output,
                                const float* fwd_out, int32_t* log, int64_t capacity_chunks,
                                int64_t chunks_used, int n_parts, float* grad_data_out,
                                void* stream, void** job_out) {
    if (!job_out) return SVOXB_ERR_NULL;
    *job_out = nullptr;
    int st = validate_tree(tree);
    if (st) return st;
    if ((st = validate_options(tree, *opt))) return st;
    if (!log || !grad_data_out || (Q > 0 && (!grad_output || !fwd_out))) return SVOXB_ERR_NULL;
    if ((st = log_eligible(tree, opt, grad_data_out))) return st;
    RenderCall c{tree, *opt, Q};
    c.backward = true;
    c.grad_out = grad_output;
    c.fwd_out = fwd_out;
    c.grad_data = grad_data_out;
    c.stream = (cudaStream_t)stream;
    c.log = log;
    c.log_capacity = capacity_chunks;
    const bool known = chunks_used > 0 && chunks_used <= capacity_chunks;
    if (!known) chunks_used = capacity_chunks;
    if (Q == 0) chunks_used = 0;
    ReplayJob* job = new (std::nothrow) ReplayJob;
    if (!job) return SVOXB_ERR_TOO_LARGE;
    st = replay_job(c, chunks_used, n_parts, job);
    if (st == SVOXB_OK && !known && Q > 0) {
        // the fallback for an overflowed log goes BEFORE the parts: if it runs, it produces the
        // whole gradient and the parts add nothing, so every part's rows are final when the
        // caller hands them on, whichever of the two happened
        c.log = nullptr;
        c.gate = LogGate{log, capacity_chunks};
        st = render_dispatch(c, src);
    }
    if (st != SVOXB_OK) {
        delete job;
        return st;
    }
    *job_out = job;
    return SVOXB_OK;
}

extern "C" {

int svoxb_replay_begin(const svoxb_tree* tree, const svoxb_rays* rays,
                       const svoxb_render_options* opt, const float* grad_output,
                       const float* fwd_out, int32_t* log, int64_t capacity_chunks,
                       int64_t chunks_used, int n_parts, float* grad_data_out, void* stream,
                       void** job) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    return replay_begin_checked(tree, RayBatch{rays->origins, rays->dirs, rays->vdirs}, rays->Q,
                                opt, grad_output, fwd_out, log, capacity_chunks, chunks_used,
                                n_parts, grad_data_out, stream, job);
}

int svoxb_replay_image_begin(const svoxb_tree* tree, const svoxb_camera* cam,
                             const svoxb_render_options* opt, const float* grad_output,
                             const float* fwd_out, int32_t* log, int64_t capacity_chunks,
                             int64_t chunks_used, int n_parts, float* grad_data_out,
                             void* stream, void** job) {
    if (!tree || !cam || !opt || !cam->c2w) return SVOXB_ERR_NULL;
    if (cam->width < 0 || cam->height < 0) return SVOXB_ERR_SHAPE;
    return replay_begin_checked(tree,
                                PixelRays{cam->c2w, cam->fx, cam->fy, cam->width, cam->height},
                                (int64_t)cam->width * cam->height, opt, grad_output, fwd_out, log,
                                capacity_chunks, chunks_used, n_parts, grad_data_out, stream, job);
}

int svoxb_replay_bin_shift(int64_t M, int32_t K) {
    if (M < 1 || K < 1) return 0;
    return replay_bin_shift(M, K);
}

int svoxb_replay_part_range(const void* job, int part, int64_t* slot_begin, int64_t* slot_end) {
    if (!job || !slot_begin || !slot_end) return SVOXB_ERR_NULL;
    const ReplayJob* j = static_cast<const ReplayJob*>(job);
    if (part < 0 || part >= j->n_parts) return SVOXB_ERR_OPTION;
    const int64_t lo = (int64_t)replay_part_first_bin(part, j->n_parts, j->n_bins) << j->shift;
    int64_t hi = (int64_t)replay_part_first_bin(part + 1, j->n_parts, j->n_bins) << j->shift;
    if (hi > j->n_slots) hi = j->n_slots;
    *slot_begin = lo < j->n_slots ? lo : j->n_slots;
    *slot_end = hi;
    return SVOXB_OK;
}

int svoxb_replay_scatter(const void* job, int part, float* grad_data_out, int reserve_sms,
                         void* stream) {
    if (!job || !grad_data_out) return SVOXB_ERR_NULL;
    ReplayJob j = *static_cast<const ReplayJob*>(job);
    if (j.tree.K % 4 == 0 && (uintptr_t)grad_data_out % 16 != 0) return SVOXB_ERR_FORMAT;
    j.to.grad = grad_data_out;
    return replay_scatter(j, part, reserve_sms, (cudaStream_t)stream);
}

int svoxb_replay_end(void* job, void*) {
    if (!job) return SVOXB_ERR_NULL;
    delete static_cast<ReplayJob*>(job);
    return SVOXB_OK;
}

int svoxb_item_log_used(const int32_t* log, int64_t* chunks_used, void* stream) {
    if (!log || !chunks_used) return SVOXB_ERR_NULL;
    int32_t head[kLogGivenUp + 1] = {0};
    SVOXB_CUDA(cudaMemcpyAsync(head, log, sizeof head, cudaMemcpyDeviceToHost,
                               (cudaStream_t)stream));
    SVOXB_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    *chunks_used = head[kLogGivenUp] != 0 ? INT64_MAX : head[0];
    return SVOXB_OK;
}

int svoxb_item_log_watch(const int32_t* log, int32_t* counts, void* stream) {
    if (!log || !counts) return SVOXB_ERR_NULL;
    SVOXB_CUDA(cudaMemcpyAsync(counts, log, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost,
                               (cudaStream_t)stream));
    return SVOXB_OK;
}

int svoxb_march_stats(const svoxb_tree* tree, const svoxb_rays* rays,
                      const svoxb_render_options* opt, int32_t* visits, int32_t* contrib_fwd,
                      int32_t* contrib_bwd, void* stream) {
    if (!tree || !rays || !opt) return SVOXB_ERR_NULL;
    if (rays->Q > 0 && (!rays->origins || !rays->dirs || !rays->vdirs)) return SVOXB_ERR_NULL;
    int st = validate_tree(tree);
    if (st) return st;
    if (!(opt->step_size >= 0.f)) return SVOXB_ERR_OPTION;
    if (rays->Q < 0) return SVOXB_ERR_SHAPE;
    if (rays->Q == 0) return SVOXB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    TopScratch scratch;
    if ((st = scratch.build(tree, 4, s))) return st;
    const TopTable top{scratch.cells, scratch.level};
    const bool in_smem = scratch.level > 0;
    const size_t smem = in_smem ? ((size_t)4 << (3 * scratch.level)) : 0;
    auto k = march_stats_kernel<256, RayBatch>;
    unsigned grid = 1;
    if ((st = persistent_grid(k, 256, smem, (rays->Q + 31) / 32, &grid))) return st;
    k<<<grid, 256, smem, s>>>(tree_args(tree), RayBatch{rays->origins, rays->dirs, rays->vdirs},
                             *opt, top, in_smem, visits, contrib_fwd, contrib_bwd, rays->Q);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

int svoxb_device_status(int clear, void* stream) {
    int word = 0;
    SVOXB_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    SVOXB_CUDA(cudaMemcpyFromSymbol(&word, g_status, sizeof(int)));
    if (clear && word != 0) {
        const int zero = 0;
        SVOXB_CUDA(cudaMemcpyToSymbol(g_status, &zero, sizeof(int)));
    }
    return word;
}

const char* svoxb_strerror(int status) {
    switch (status) {
        case SVOXB_OK: return "ok";
        case SVOXB_ERR_NULL: return "a required pointer is null";
        case SVOXB_ERR_SHAPE: return "inconsistent or negative size";
        case SVOXB_ERR_FORMAT: return "data format / record layout not supported";
        case SVOXB_ERR_OPTION: return "invalid render option";
        case SVOXB_ERR_CUDA: return "CUDA runtime error";
        case SVOXB_ERR_TREE: return "corrupt tree: a descent left the node array";
        case SVOXB_ERR_MARCH: return "a ray exceeded the marching step cap";
        case SVOXB_ERR_TOO_LARGE: return "size beyond the supported maximum";
    }
    return "unknown status";
}

const char* svoxb_last_cuda_error(void) { return t_cuda_error; }

int svoxb_reserve_sms(int n) {
    const int before = g_reserved_sms;
    if (n >= 0) g_reserved_sms = n;
    return before;
}

int svoxb_allreduce_multimem(float* multicast, int64_t n_floats, int rank, int world,
                             void* stream) {
    if (!multicast) return SVOXB_ERR_NULL;
    if (world < 1 || rank < 0 || rank >= world || n_floats < 0) return SVOXB_ERR_OPTION;
    if ((uintptr_t)multicast % 16 != 0 || n_floats % 4 != 0) return SVOXB_ERR_SHAPE;
    const int64_t words = n_floats / 4;
    const int64_t first = words * rank / world, last = words * (rank + 1) / world;
    if (last <= first) return SVOXB_OK;
    int sms = sm_count() - g_reserved_sms;
    if (sms < 1) sms = 1;
    int64_t grid = (last - first + kReduceBlock - 1) / kReduceBlock;
    if (grid > 2 * sms) grid = 2 * sms;
    multimem_allreduce_kernel<<<(unsigned)grid, kReduceBlock, 0, (cudaStream_t)stream>>>(
        multicast, first, last);
    SVOXB_CUDA(cudaGetLastError());
    return SVOXB_OK;
}

const char* svoxb_version(void) { return "0.4.5"; }

// Test hook (include/svox_b200_testing.h): key 5 = MB of gradient one replay bin spans,
// key 7 = bricks below the render leaf table on / off.
int svoxb_test_knob(int key, int value) {
    switch (key) {
        case 7: g_tuning.render_bricks = value != 0; return SVOXB_OK;
        case 5:
            if (value < 1 || value > 1024) return SVOXB_ERR_OPTION;
            g_tuning.replay_bin_mb = value;
            return SVOXB_OK;
    }
    return SVOXB_ERR_OPTION;
}

int svoxb_test_known_launches(void) {
    std::lock_guard<std::mutex> lock(g_known_mutex);
    return (int)g_known.size();
}

}  // extern "C"

#include "noalloc.cuh"
