// Backward march: the gradient of a render without an item log, and the fallback for a log that cannot
// be replayed (render_replay.cuh).  The forward's design (render_queue.cuh: G and S steps, queue,
// staging rows, refills), in one march when the forward's result is given, else in two.  In the S
// step lane i forms the gradient of record i in its staging row and the warp flushes the rows with
// red.global.add.v4.f32, 16 bytes per lane.
//
// The march is the forward's as it was before that was shortened further.  A trial of the shorter form in
// here ended in an illegal instruction, in a test that launches the plain forward and then this
// kernel; which of the two raised it was not established, and no cause was found by reading.
#pragma once

#include "render_queue.cuh"

namespace svoxb {

// Shared memory of one warp.
template <int BD>
struct alignas(16) BackQueue {
    static constexpr int K = RecordLength<BD>::K;
    using Shape = RecordShape<K>;
    static constexpr int CAP = 64;     // two batches: items being collected, and what spills over
    // per ray: colour basis, upstream gradient, delta_scale; odd stride: no bank conflicts
    static constexpr int SCALE = BD + 3;
    static constexpr int RAYW = (SCALE + 1) | 1;
    // Staging rows (cp.async targets).  After lane i has read row i it reuses the
    // row's first words for the item's results.
    alignas(16) float rows[32 * Shape::STRIDE];
    uint32_t slot[CAP];
    float dt[CAP];                     // step length
    float sigma[CAP];
    unsigned char owner[CAP];          // bits 0-4 owner lane, bit 7 accumulation march
    float rayv[32][RAYW];
};

template <int BD>
constexpr int back_blocks_per_sm() {
    const int fit = (int)(227 * 1024 / ((kMarchBlock / 32) * sizeof(BackQueue<BD>) + 1024));
    return fit > kMarchBlocks ? kMarchBlocks : fit < 1 ? 1 : fit;
}

template <int BD, class Source>
__global__ void __launch_bounds__(kMarchBlock, back_blocks_per_sm<BD>())
render_back_kernel(TreeArgs tr, Source src, svoxb_render_options opt, TreeIndex index,
                   int64_t tickets, const float* __restrict__ grad_out,
                   const float* __restrict__ fwd_out, float* __restrict__ grad_data, LogGate gate,
                   MarchShape shape) {
    constexpr int K = RecordLength<BD>::K;
    using WQ = BackQueue<BD>;
    using Shape = RecordShape<K>;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ unsigned s_next;
    // with a log: the marching fallback of a replay, for a log that is not complete
    if (gate.closed()) return;
    if (threadIdx.x == 0) s_next = 0;
    const int lane = threadIdx.x & 31;
    WQ& q = *reinterpret_cast<WQ*>(s_raw + (size_t)(threadIdx.x >> 5) * sizeof(WQ));
    __syncthreads();
    const float d_rgb_pad = 1 + 2 * opt.rgb_padding;
    const bool single = fwd_out != nullptr;
    const float bg = opt.background_brightness;
    const int L = index.level;
    const uint32_t side = (1u << L) - 1u;
    const uint64_t pol_keep = l2_policy_keep(), pol_stream = l2_policy_stream();
    const bool vec_ok = (reinterpret_cast<uintptr_t>(grad_data) & 15) == 0;

    // ---- per-lane state -------------------------------------------------------
    Ray r{};        // (lanes without a ray compute along)
    int64_t ray = 0;
    int state = lane < shape.lanes ? kNeedRay : kExhausted;
    float t = 0.f, light = 1.f;   // transmittance after the items folded
    float accum = 0.f;
    int phase = 1;  // 0 = accumulation march (reference PASS 1), 1 = scatter march
    int it = 0;
    uint32_t cur_cell = 0xffffffffu;   // table cell of the brick used last ...
    uint32_t cur_brick = 0;            // ... and where the brick lies in the index
    // cursor: the position of the lane's next sample, and the index words requested for it
    float px = 0.f, py = 0.f, pz = 0.f;
    int2 entry = make_int2(0, 0);
    uint32_t cell = 0;                 // ... and its table cell
    bool in_brick = false;             // ... from the brick `cur_brick`, else from the table
    // queue: ring of two batches; `qn` items collected from ring position `head` on
    int head = 0, qn = 0;
    unsigned mine = 0u, mine_next = 0u, mine_fly = 0u;  // my items: first 32, spilled, in flight
    int fly = 0;                       // items in flight; this lane's:
    uint32_t fly_slot = 0u;
    float fly_dt = 0.f, fly_sigma = 0.f;
    int fly_own = 0;

    // Places the cursor at parameter t and requests the index words there, to be consumed one
    // iteration later: the brick's, if the ray is still in the table cell whose brick it used
    // last, else the table's.
    auto place_cursor = [&]() {
        px = fminf(__saturatef(mad_site<FC_POS>(t, r.dx, r.ox)), kPosMax);
        py = fminf(__saturatef(mad_site<FC_POS>(t, r.dy, r.oy)), kPosMax);
        pz = fminf(__saturatef(mad_site<FC_POS>(t, r.dz, r.oz)), kPosMax);
    };
    // 1 + floor(p * 2^23) / 2^23, exactly: the low 23 bits are the position's bits
    auto bits = [](float p) { return __float_as_uint(__fadd_rz(p, 1.0f)); };
    auto request_words = [&]() {
        const uint32_t ux = bits(px), uy = bits(py), uz = bits(pz);
        if (index.table == nullptr) {       // fallback march: no index was built
            entry = make_int2(kWordWalk, 0);
            in_brick = false;
            return;
        }
        cell = ((ux >> (kPosBits - 3 * L)) & (side << (2 * L))) |
               ((uy >> (kPosBits - 2 * L)) & (side << L)) | ((uz >> (kPosBits - L)) & side);
        in_brick = cell == cur_cell;
        const int s3 = kPosBits - kBrickLevels - L;
        const uint32_t c = ((ux >> (s3 - 6)) & 0x1c0u) | ((uy >> (s3 - 3)) & 0x38u) |
                           ((uz >> s3) & 7u);
        entry = ld_keep(index.table + (in_brick ? cur_brick + c : cell), pol_keep);
    };

    // Takes the first n (<= 32) collected items as the batch in flight and requests their
    // records: consecutive lanes copy consecutive 16-byte words, asynchronously.
    auto request = [&](int n) {
        fly_slot = q.slot[head + lane];
        fly_dt = q.dt[head + lane];
        fly_sigma = q.sigma[head + lane];
        fly_own = q.owner[head + lane];
        const uint32_t slot = lane < n ? fly_slot : 0u;
        mine_fly = mine;
        mine = mine_next;
        mine_next = 0u;
        fly = n;
        head ^= 32;
        qn = qn > 32 ? qn - 32 : 0;
        const int sub = lane / Shape::GROUP, w = lane % Shape::GROUP;
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
        const uint32_t b_slot = fly_slot;
        const int b_own = fly_own;
        float* row = q.rows + lane * Shape::STRIDE;
        const int off = record_offset<K>(tr.data, b_slot);
        const int own = b_own & 31;
        const bool acc_item = (b_own & 0x80) != 0;
        float sg[3] = {0.f, 0.f, 0.f}, col[3] = {0.f, 0.f, 0.f};
        float raw_sigma = 0.f, att = 0.f, b_dd = 0.f;
        if (active) {
            const float delta_t = fly_dt, sigma = fly_sigma,
                        delta_scale = q.rayv[own][WQ::SCALE];
            b_dd = delta_t * delta_scale;
            att = expf(-delta_t * sigma * delta_scale);
            float tmp[3] = {0.f, 0.f, 0.f};
            if (BD == 0) {
                const float4 x = *reinterpret_cast<const float4*>(row);
                tmp[0] = x.x; tmp[1] = x.y; tmp[2] = x.z;
                raw_sigma = x.w;
            } else {
                float bs[BD > 0 ? BD : 1];
#pragma unroll
                for (int i = 0; i < BD; ++i)
                    if (Shape::ALIGNED) bs[i] = q.rayv[own][i];
                if (Shape::ALIGNED) {
#pragma unroll
                    for (int w = 0; w < K / 4; ++w) {
                        const float4 x = reinterpret_cast<const float4*>(row)[w];
                        const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int e = 4 * w + i;
                            if (e < K - 1)
                                tmp[e / (BD > 0 ? BD : 1)] = __fmaf_rn(
                                    bs[e % (BD > 0 ? BD : 1)], v[i], tmp[e / (BD > 0 ? BD : 1)]);
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
#pragma unroll
                    for (int m = 0; m < B; ++m)
                        bs[m] = q.rayv[own][m >= 3 || m >= off ? m - off : m - off + B];
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
            }
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                sg[ch] = sigmoid_ref(tmp[ch]);
                col[ch] = sg[ch] * d_rgb_pad - opt.rgb_padding;
            }
            float total_color = 0.f;
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) total_color += col[ch] * q.rayv[own][BD + ch];
            *reinterpret_cast<float4*>(row) =
                make_float4(total_color, att, acc_item ? 1.f : 0.f, b_dd);
        }
        __syncwarp();
        // every owner folds in its items, in march order
        for (unsigned m = mine_fly; m != 0u; m &= m - 1u) {
            float4* res = reinterpret_cast<float4*>(q.rows + (__ffs(m) - 1) * Shape::STRIDE);
            const float4 x = *res;
            const float weight = light * (1.f - x.y);
            light = light * x.y;
            if (x.z != 0.f) {
                accum += weight * x.x;
            } else {
                accum -= weight * x.x;
                res->x = x.w * (x.x * light - accum);    // density gradient
                res->y = weight;
            }
        }
        mine_fly = 0u;
        fly = 0;
        __syncwarp();
        // lane i forms the gradient of record i in its staging row
        const int goff = record_offset<K>(grad_data, b_slot);
        if (active && !acc_item) {
            const float gs = row[0], b_w = row[1];
            float v[K];
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                const float tmp2 = b_w * sg[ch] * (1.0 - sg[ch]) * q.rayv[own][BD + ch] *
                                   d_rgb_pad;
                if (BD == 0) v[ch] = tmp2;
#pragma unroll
                for (int i = 0; i < BD; ++i) v[ch * BD + i] = q.rayv[own][i] * tmp2;
            }
            v[K - 1] = gs * (opt.density_softplus ? sigmoid_ref(raw_sigma - 1) : 1);
            if (Shape::ALIGNED) {
#pragma unroll
                for (int w = 0; w < K / 4; ++w)
                    reinterpret_cast<float4*>(row)[w] =
                        make_float4(v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 3; ++i) {       // the row's places around the record
                    if (i < goff) row[i] = 0.f;
                    if (goff + K + i < 4 * Shape::WORDS) row[goff + K + i] = 0.f;
                }
#pragma unroll
                for (int w = 0; w < K; ++w) row[goff + w] = v[w];
            }
        }
        __syncwarp();
        const int sub = lane / Shape::GROUP, w = lane % Shape::GROUP;
        const int meta = goff | (acc_item ? 8 : 0);
#pragma unroll
        for (int p = 0; p < Shape::GROUP; ++p) {
            const int k = p * Shape::RPP + sub;
            const uint32_t s = __shfl_sync(0xffffffffu, b_slot, k);
            const int m = __shfl_sync(0xffffffffu, meta, k);
            if (k < nb && w < Shape::WORDS && m < 8)
                flush_word<K>(grad_data + (size_t)s * K, m & 3, w,
                              reinterpret_cast<const float4*>(q.rows + k * Shape::STRIDE)[w],
                              vec_ok, pol_stream);
        }
        __syncwarp();
    };

    unsigned alive = __ballot_sync(0xffffffffu, state != kExhausted);
    for (;;) {
        // ---- lanes that are not marching: finish, refill, termination ---------------------
        unsigned marching = __ballot_sync(0xffffffffu, state == kMarching);
        const unsigned waiting = alive & ~marching;
        if (marching == 0u || __popc(waiting) >= shape.refill) {
            if (__any_sync(0xffffffffu, state == kEnded && (mine | mine_next | mine_fly) != 0u)) {
                __syncwarp();
                if (fly > 0) evaluate();
                while (qn > 0) {
                    request(qn < 32 ? qn : 32);
                    evaluate();
                }
            }
            if (state == kEnded) {
                state = kNeedRay;
                if (phase == 0) {
                    // tail of the reference's PASS 1 (rt_kernel.cu:415-418), then march again
                    const float* g = &q.rayv[lane][BD];
                    const float total_grad = g[0] + g[1] + g[2];
                    accum += light * bg * total_grad;
                    phase = 1;
                    t = r.tmin; light = 1.f; it = 0;
                    state = kMarching;
                    place_cursor();
                    request_words();
                }
            }
            if (state == kNeedRay) {
                const unsigned ticket = atomicAdd(&s_next, 1u);
                const int gs = shape.granule_shift;
                const int64_t first =
                    ((int64_t)blockIdx.x + (int64_t)gridDim.x * (ticket >> gs)) << gs;
                const int64_t place = first + (ticket & ((1u << gs) - 1u));
                if (first >= tickets) {
                    state = kExhausted;
                } else if (place < tickets && (ray = src.pick(place)) >= 0) {
                    src.load(ray, tr, opt, r);
                    ray_setup(r, tr.scaling);
                    if (r.hit && r.tmin < r.tmax) {
                        march_ready(r);
                        state = kMarching;
                        t = r.tmin; light = 1.f; it = 0;
                        q.rayv[lane][WQ::SCALE] = r.delta_scale;
                        place_cursor();
                        request_words();
                        if (BD > 0) {
                            float basis[BD > 0 ? BD : 1];
                            colour_basis<(BD > 0 ? BD : 1), Source::kLobes>(tr, opt, r.vdir, basis);
#pragma unroll
                            for (int i = 0; i < BD; ++i)
                                q.rayv[lane][i] =
                                    (i < opt.min_comp || i > opt.max_comp) ? 0.f : basis[i];
                        }
                        const float g0 = __ldg(grad_out + 3 * ray), g1 = __ldg(grad_out + 3 * ray + 1),
                                    g2 = __ldg(grad_out + 3 * ray + 2);
                        float* g = &q.rayv[lane][BD];
                        g[0] = g0; g[1] = g1; g[2] = g2;
                        accum = 0.f;
                        phase = single ? 1 : 0;
                        if (single) {
                            accum = __ldg(fwd_out + 3 * ray) * g0;
                            accum += __ldg(fwd_out + 3 * ray + 1) * g1;
                            accum += __ldg(fwd_out + 3 * ray + 2) * g2;
                        }
                    }
                }
            }
            __syncwarp();
            marching = __ballot_sync(0xffffffffu, state == kMarching);
            alive = __ballot_sync(0xffffffffu, state != kExhausted);
            if (marching == 0u) {
                if (alive == 0u) break;
                continue;
            }
        }

        // ---- G step: every lane consumes the words requested one iteration ago --------------
        // (without branches but for the rare cases: lanes that have nothing to do compute along)
        bool on = state == kMarching;
        if (on && !in_brick && entry.x < 0) {
            // the table cell has a brick: the sample is looked up there
            cur_cell = cell;
            cur_brick = index.bricks + (uint32_t)(entry.x & 0x7fffffff) * kBrickCells;
            on = false;
        }
        uint32_t slot = (uint32_t)entry.y & 0x0fffffffu;
        float sigma = __int_as_float(entry.x);
        bool item = on && entry.x <= kWordInf;      // the leaf passes the density test
        bool done = false;
        // side of the leaf's cube, 2^-depth
        float inv_cube = __int_as_float((127 << 23) - (int)((uint32_t)entry.y >> 28 << 23));
        float fine = 0.f;
        if (on && entry.x >= kWordFetch) {
            // seldom: a tree deeper than the index, a density that is not in the word
            float raw = 0.f;
            if (entry.x == kWordWalk) {
                const float big = (float)(1 << 24);
                const int depth = (int)((uint32_t)entry.y >> 28);
                const Walked f = walk_to_leaf(
                    tr.child, tr.data, K, tr.M, depth > L ? (int64_t)slot : 0,
                    depth > L ? depth - 1 : 0, (int)(px * big), (int)(py * big), (int)(pz * big));
                done = !f.ok;
                if (done) report(SVOXB_ERR_TREE);
                slot = f.slot;
                inv_cube = __int_as_float((127 - (f.ok ? f.depth : 1)) << 23);
                raw = f.raw;
                // 2^-24 leaves: a float resolves them below 1/2, where the sum below would not
                if (f.ok && f.depth > kPosBits) fine = 1.f;
            } else {
                raw = __ldg(tr.data + (size_t)slot * K + (K - 1));
            }
            sigma = opt.density_softplus ? softplus_m1(raw) : raw;
            item = !done && sigma > 0.f;
        }
        // Lower corner of the leaf: a number whose last place is the leaf's side takes in the
        // position's multiples of it and drops the rest.
        const float coarse = __int_as_float(__float_as_int(inv_cube) + (kPosBits << 23));
        float cx = __fsub_rn(__fadd_rz(px, coarse), coarse);
        float cy = __fsub_rn(__fadd_rz(py, coarse), coarse);
        float cz = __fsub_rn(__fadd_rz(pz, coarse), coarse);
        if (fine != 0.f) {
            const float big = (float)(1 << 24);
            cx = truncf(px * big) * (1.f / big);
            cy = truncf(py * big) * (1.f / big);
            cz = truncf(pz * big) * (1.f / big);
        }
        // Exit distance of the leaf (_dda_unit, svox/csrc/rt_kernel.cu:203-220, in the leaf's own
        // scale).  The point lies inside, so the entry distance is 0 and per axis the larger of
        // t1 = -f*inv and t1 + inv is t1 + max(inv, 0); powers of two commute with rounding, so
        // everything can be done at the tree's scale.
        const float ex = __fmaf_rn(fmaxf(r.ix, 0.f), inv_cube,
                                   __fmul_rn(__fsub_rn(cx, px), r.ix));
        const float ey = __fmaf_rn(fmaxf(r.iy, 0.f), inv_cube,
                                   __fmul_rn(__fsub_rn(cy, py), r.iy));
        const float ez = __fmaf_rn(fmaxf(r.iz, 0.f), inv_cube,
                                   __fmul_rn(__fsub_rn(cz, pz), r.iz));
        const float delta_t = __fadd_rn(fminf(ex, fminf(ey, ez)), opt.step_size);
        if (on) {
            t = __fadd_rn(t, delta_t);
            if (!(t < r.tmax)) done = true;
            if (++it > kMaxSteps) {
                report(SVOXB_ERR_MARCH);
                done = true;
            }
            if (done) state = kEnded;
        }
        place_cursor();
        if (state == kMarching) request_words();

        // ---- push items --------------------------------------------------------------
        const unsigned pushed = __ballot_sync(0xffffffffu, item);
        if (item) {
            const int n = qn + __popc(pushed & ((1u << lane) - 1u));
            const int pos = (head + n) & (WQ::CAP - 1);
            q.slot[pos] = slot;
            q.dt[pos] = delta_t;
            q.sigma[pos] = sigma;
            q.owner[pos] = (unsigned char)(lane | (phase == 0 ? 0x80 : 0));
            const unsigned bit = 1u << (n & 31);
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

}  // namespace svoxb
