"""The branches that a call's size, record length or history selects, at the sizes where they
begin and end: each against the branch beside it, the definition in torch, or the marching
backward.  Needs a GPU."""
import numpy as np
import pytest
import torch

import svox_b200 as svox
from svox_b200 import csrc, render as _render
from svox_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _shell(fmt, refine, extra, dev, seed=5):
    gen = torch.Generator().manual_seed(seed)
    return W.shell_tree(refine, extra, fmt, gen, (5.0, 50.0), W._SHELL).to(dev)


def _rays(n, dev, seed=6):
    gen = torch.Generator().manual_seed(seed)
    return svox.Rays(*[t.to(dev) for t in W.sphere_rays(n, gen, 4.0, 0.2, 0.8)])


def _close(a, b):
    # sums of the same 32-bit terms in another order: 1e-5 of the largest element, the bound that
    # the reference's own two runs of a backward keep (parity_util.assert_grad_matches_reference)
    return (a - b).abs().max().item() <= 1e-5 * b.abs().max().item()


def _grad(renderer, call, upstream):
    renderer.tree.data.grad = None
    call().backward(upstream)
    return renderer.tree.data.grad


@pytest.fixture(scope="module")
def big_tree(cuda_device):
    """512^3 shell of 1.3 M nodes with the shortest records (large enough for bricks only where
    the rays pass)."""
    return _shell("SH1", 5, 3, cuda_device)


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024])
def test_bricks_where_a_few_rays_pass(n, big_tree, cuda_device):
    r = svox.VolumeRenderer(big_tree)
    rays = _rays(2048, cuda_device)                      # more rays: every brick
    with torch.no_grad():
        every = r(rays)
        some = r(svox.Rays(*[t[:n].contiguous() for t in rays]))
    assert torch.equal(some, every[:n])
    csrc.check_device_status()


@pytest.mark.parametrize("fmt", ["RGBA", "SH4", "SH9", "SH16"])
def test_few_rays_and_many_give_the_same(fmt, cuda_device):
    # up to 16 warps of rays per SM go through smaller blocks, compiled for fewer of them
    r = svox.VolumeRenderer(_shell(fmt, 3, 2, cuda_device))
    few = torch.cuda.get_device_properties(cuda_device).multi_processor_count * 512
    rays = _rays(few + 33, cuda_device)
    with torch.no_grad():
        every = r(rays)
        for n in (few, 4097, 33):
            assert torch.equal(r(svox.Rays(*[t[:n].contiguous() for t in rays])), every[:n])
    csrc.check_device_status()


@pytest.mark.parametrize("thresh", [1e-40, 1e-30, 1e-2, 0.5, 0.97, 1.0, 3.0, float("inf")])
@pytest.mark.parametrize("fmt", ["RGBA", "SH9"])
def test_early_stop_against_the_kernel_that_multiplies_as_it_goes(fmt, thresh, cuda_device):
    # The march ends a ray by its summed optical depth, the evaluation by the product of its
    # attenuations; records at odd addresses take the one-thread-per-ray kernel, which stops by the
    # same product.  Many rays cross empty space first, where nothing may stop them.
    tree = _shell(fmt, 3, 3, cuda_device)
    tree.data.data[..., -1] *= 8.0
    tree.data.requires_grad_(False)
    rays = _rays(5003, cuda_device)
    r = svox.VolumeRenderer(tree)
    r.stop_thresh = thresh
    out = r(rays)
    odd = torch.empty(tree.data.numel() + 1, device=cuda_device)[1:].view(tree.data.shape)
    odd.copy_(tree.data)
    tree.data.data = odd
    want = r(rays)
    # (rounding of the colours' sums: the stop itself is the same bits.  What the small thresholds leave
    # changes no colour: test_early_stop_leaf_by_leaf tells where those stop.)
    assert (out - want).abs().max().item() <= 1e-5
    csrc.check_device_status()


@pytest.mark.parametrize("op", ["sum", "max"])
def test_weights_of_rays_that_stop_early(op, cuda_device):
    # samples that the march still took behind a ray's stop leave no weight
    tree = _shell("RGBA", 3, 3, cuda_device)
    tree.data.data[..., -1] *= 8.0
    tree.data.requires_grad_(False)
    rays = _rays(5003, cuda_device)
    r = svox.VolumeRenderer(tree)
    r.stop_thresh = 0.3

    def weights():
        with tree.accumulate_weights(op=op) as accum:
            r(rays)
        return accum()

    out = weights()
    odd = torch.empty(tree.data.numel() + 1, device=cuda_device)[1:].view(tree.data.shape)
    odd.copy_(tree.data)
    tree.data.data = odd                 # (the one-thread-per-ray kernel)
    want = weights()
    # a largest weight is the same product; sums of up to some hundred weights in another order
    if op == "max":
        assert torch.equal(out, want)
    else:
        assert _close(out, want)
    csrc.check_device_status()


def _eight_leaves(fmt, sigma, dev):
    """A tree of one node; density of the half x > 1/2."""
    tree = svox.N3Tree(N=2, data_format=fmt, init_refine=0, device=dev)
    tree.data.data.fill_(0.3)
    tree.data.data[..., -1] = 0.0
    tree.data.data[0, 1, :, :, -1] = sigma
    return tree


def _along_x(n, sign, dev, seed=3):
    """Parallel rays along the axis x through both halves of the unit cube."""
    yz = torch.rand(n, 2, generator=torch.Generator().manual_seed(seed)) * 0.4 + 0.05
    origins = torch.cat((torch.full((n, 1), 0.5 - 2.0 * sign), yz), 1).to(dev)
    dirs = torch.tensor([[float(sign), 0.0, 0.0]]).expand(n, 3).contiguous().to(dev)
    return svox.Rays(origins, dirs, dirs.clone())


@pytest.mark.parametrize("what,code", [("damaged", 6), ("stuck", 7)])
@pytest.mark.parametrize("fmt", ["RGBA", "SH9", "SH25"])
def test_nothing_behind_an_early_stop_is_reported(fmt, what, code, cuda_device):
    # The first half has an optical depth of 0.72: exp(-0.72) = 0.487.  Behind it lies a node that
    # does not exist, or (step size 0) the rays do not get off its far side, which has an extent
    # of 0 in their direction.
    tree = _eight_leaves(fmt, 1.44, cuda_device)
    tree.data.requires_grad_(False)
    if what == "damaged":
        tree.child[0, 0, 0, 0] = 1_000_000
    r = svox.VolumeRenderer(tree, step_size=1e-3 if what == "damaged" else 0.0)
    rays = _along_x(37, -1, cuda_device)
    r.stop_thresh = 0.5
    out = r(rays)
    assert csrc.device_status(clear=True) == 0
    if fmt == "RGBA":                       # the colour of what was met, whatever its weight
        assert (out - torch.sigmoid(torch.tensor(0.3))).abs().max().item() < 1e-5
    r.stop_thresh = 0.48                    # not reached
    r(rays)
    assert csrc.device_status(clear=True) == code


def _at_odd_addresses(tree):
    """The tree's records where only the one-thread-per-ray kernels take them."""
    odd = torch.empty(tree.data.numel() + 1, device=tree.data.device)[1:].view(tree.data.shape)
    odd.copy_(tree.data)
    tree.data.data = odd


def _largest_weights(tree, renderer, rays):
    with torch.no_grad(), tree.accumulate_weights(op="max") as accum:
        renderer(rays)
    return accum()


def test_early_stop_among_negative_densities(cuda_device):
    # Four leaves in a row, of depth -89, 45, 46 and 1.  The transmittance overflows in the first and is
    # infinite from there on, so the ray never stops, although the depths' sum passes the
    # threshold in the third.
    tree = svox.N3Tree(N=2, data_format="RGBA", init_refine=1, device=cuda_device)
    tree.data.requires_grad_(False)
    x = torch.tensor([0.875, 0.625, 0.375, 0.125], device=cuda_device)
    depth = torch.tensor([-89.0, 45.0, 46.0, 1.0], device=cuda_device)
    points = torch.cartesian_prod(x, x, x)
    _, ids = tree(points, want_node_ids=True)
    tree.data.data.view(-1, 4)[ids, -1] = depth.repeat_interleave(16) / 0.251
    r = svox.VolumeRenderer(tree)
    r.sigma_thresh, r.stop_thresh = -1e9, 0.5
    rays = _along_x(37, -1, cuda_device)
    out = _largest_weights(tree, r, rays)
    _at_odd_addresses(tree)
    want = _largest_weights(tree, r, rays)
    last = ids[points[:, 0] == 0.125]
    assert torch.isinf(want.view(-1)[last]).any()
    assert torch.equal(out, want)
    csrc.check_device_status()


@pytest.mark.parametrize("thresh", [1e-40, 1e-30, 1e-2, 0.5])
@pytest.mark.parametrize("fmt", ["RGBA", "SH9"])
def test_early_stop_leaf_by_leaf(fmt, thresh, cuda_device):
    # 32 leaves of depth 3 to 5 in every row, each met by rays that have come through the same
    # ones: the leaves with a weight are the leaves before the stop, however small the threshold
    tree = svox.N3Tree(N=2, data_format=fmt, init_refine=4, device=cuda_device)
    tree.data.requires_grad_(False)
    gen = torch.Generator().manual_seed(4)
    sigma = (3.0 + 2.0 * torch.rand(tree.data.shape[:-1], generator=gen)) / (1 / 32 + 1e-3)
    tree.data.data[..., -1] = sigma.to(cuda_device)
    r = svox.VolumeRenderer(tree)
    rays = _along_x(2000, -1, cuda_device)
    every = _largest_weights(tree, r, rays)
    r.stop_thresh = thresh
    out = _largest_weights(tree, r, rays)
    _at_odd_addresses(tree)
    want = _largest_weights(tree, r, rays)
    assert (want > 0).sum() < (every > 0).sum()
    assert torch.equal(out, want)           # the same products
    csrc.check_device_status()


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("fmt", ["RGBA", "SH9", "SH25"])
def test_sample_cap(fmt, grad, cuda_device):
    # With a step size of 0 rays towards -x do not get off the plane x = 1/2 (see above), those towards
    # +x do.  The former end at the cap with a status; the others are what they are alone.
    tree = _eight_leaves(fmt, 1.44, cuda_device)
    tree.data.requires_grad_(grad)
    r = svox.VolumeRenderer(tree, step_size=0.0)
    good = _along_x(75, 1, cuda_device)
    want = r(good)
    assert csrc.device_status(clear=True) == 0
    bad = _along_x(5, -1, cuda_device)
    mixed = svox.Rays(*[torch.cat((a[:40], b, a[40:])) for a, b in zip(good, bad)])
    out = r(mixed)
    assert csrc.device_status(clear=True) == 7
    assert torch.equal(torch.cat((out[:40], out[45:])), want)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("fmt,refine,n_rays", [("RGBA", 5, 50000), ("SH9", 4, 12000),
                                               ("SH16", 4, 12000)])
@pytest.mark.parametrize("image", [False, True])
def test_sorted_log_unsorted_log_and_march_agree(fmt, refine, n_rays, image, cuda_device):
    # 169 k (RGBA: 1.3 M) nodes: the gradient (169, 152, 266 MB) outgrows a bin, and the rays (or
    # 400 x 300 pixels) touch enough of it for the log to be sorted and the gradient cleared on
    # the way
    tree = _shell(fmt, refine, 3, cuda_device)
    r = svox.VolumeRenderer(tree)
    if image:
        c2w = W.look_at_cameras(1, torch.Generator().manual_seed(1), 1.6)[0].to(cuda_device)

        def call():
            return r.render_persp(c2w, width=400, height=300, fx=560.0)
    else:
        rays = _rays(n_rays, cuda_device)

        def call():
            return r(rays)
    up = torch.randn(call().shape, generator=torch.Generator(cuda_device).manual_seed(2),
                     device=cuda_device)
    n = up.numel() // 3
    lib = csrc.library()
    assert csrc.log_is_sorted(tree._spec(), n, image)
    a = _grad(r, call, up)
    try:
        assert lib.svoxb_test_knob(5, 1024) == 0         # one bin: nothing to sort
        assert not csrc.log_is_sorted(tree._spec(), n, image)
        b = _grad(r, call, up)
    finally:
        lib.svoxb_test_knob(5, 32)
    _render.USE_ITEM_LOG = False
    try:
        c = _grad(r, call, up)
    finally:
        _render.USE_ITEM_LOG = True
    assert _close(a, c) and _close(b, c)
    csrc.check_device_status()


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("n", [1, 37, 4097])
@pytest.mark.parametrize("fmt", ["RGBA", "SH9", "SH16"])
def test_marching_backward_with_lanes_that_have_no_ray(fmt, n, two, cuda_device):
    # warps with fewer rays than lanes, and rays that miss the cube among them: those lanes compute along
    tree = _shell(fmt, 3, 2, cuda_device)
    r = svox.VolumeRenderer(tree)
    origins, dirs, views = _rays(n, cuda_device)
    origins[1::5] += 40.0
    rays = svox.Rays(origins, dirs, views)
    up = torch.randn(n, 3, generator=torch.Generator().manual_seed(2)).to(cuda_device)
    a = _grad(r, lambda: r(rays), up)
    _render.USE_ITEM_LOG, _render.FORCE_TWO_MARCHES = False, two
    try:
        b = _grad(r, lambda: r(rays), up)
    finally:
        _render.USE_ITEM_LOG, _render.FORCE_TWO_MARCHES = True, False
    assert b.abs().max().item() > 0
    assert _close(b, a)
    csrc.check_device_status()


@pytest.mark.parametrize("fmt", ["RGBA", "SH4"])
@pytest.mark.parametrize("n", [50, 30000])
def test_se_grad_through_either_log_and_without(fmt, n, cuda_device):
    # few rays: unsorted log, results cleared beside the march; many: sorted; a log that is too
    # small: the march enqueued behind the replay
    tree = _shell(fmt, 4, 3, cuda_device)
    r = svox.VolumeRenderer(tree)
    rays = _rays(n, cuda_device)
    colors = torch.rand(n, 3, generator=torch.Generator(cuda_device).manual_seed(3),
                        device=cuda_device)
    out, grad, hess = r.se_grad(rays, colors)
    old = csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS
    csrc.log_estimate(wait=True)
    try:
        csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS = 0.0, 2
        out2, grad2, hess2 = r.se_grad(rays, colors)
        csrc.log_estimate(wait=True)
        assert csrc._LogWatch.last_used > csrc._LogWatch.last_cap
    finally:
        csrc.log_estimate(wait=True)
        csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS = old
    assert torch.equal(out, out2)
    # the reference adds the density's gradient once per channel, the replay the channels' sum:
    # 3e-4 of the summed magnitude in the parity tests, of the largest element here
    assert (grad - grad2).abs().max() <= 3e-4 * grad2.abs().max()
    assert (hess - hess2).abs().max() <= 3e-4 * hess2.abs().max()
    csrc.check_device_status()


@pytest.mark.parametrize("fmt", ["SH4", "SH16"])
@pytest.mark.parametrize("n", [200, 30000])
@pytest.mark.parametrize("at", [(0, 0), (0, 1), (2, 0), (3, 1)])
def test_se_grad_into_buffers_of_different_alignment(fmt, n, at, cuda_device):
    # both results are expanded through the same rows of shared memory, shifted to their words
    # (records of whole 16-byte words have to lie on them: SVOXB_ERR_FORMAT)
    import ctypes as C
    tree = _shell(fmt, 4, 3, cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(n, cuda_device)
    spec, src, opt = tree._spec(), _render._rays_spec_from_rays(rays), r._get_options()
    resid = torch.randn(n, 3, generator=torch.Generator(cuda_device).manual_seed(3),
                        device=cuda_device)
    r.se_grad(rays, resid)
    csrc.log_estimate(wait=True)            # the next log is large enough
    out, (log, cap) = csrc.volume_render_logged(spec, src, opt)
    used = csrc.log_chunks_used(log)
    assert used <= cap
    want = r.se_grad(rays, out - resid)[1:]
    size = tree.data.numel()
    got = [torch.full((size + 8,), float("nan"), device=cuda_device) for _ in at]
    ct, cr, co = csrc._pack_tree(spec), csrc._pack_rays(src, tree.data.device), opt._pack()
    assert csrc.library().svoxb_se_grad_replay(
        C.byref(ct), C.byref(cr), C.byref(co), C.c_void_p(resid.data_ptr()),
        C.c_void_p(out.data_ptr()), C.c_void_p(log.data_ptr()), C.c_int64(cap), C.c_int64(used),
        *[C.c_void_p(g.data_ptr() + 4 * k) for g, k in zip(got, at)], C.c_int(1),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    for g, k, w in zip(got, at, want):
        assert _close(g[k:k + size], w.reshape(-1))
        assert g[:k].isnan().all() and g[k + size:].isnan().all()
    csrc.check_device_status()


@pytest.mark.parametrize("n", [40, 12000])
def test_backward_twice_over_one_forward(n, cuda_device):
    # a gradient cleared beside the forward is handed out once; a sorted log is replayed twice
    tree = _shell("SH9", 4, 3, cuda_device)
    r = svox.VolumeRenderer(tree)
    out = r(_rays(n, cuda_device))
    up = torch.ones_like(out)
    tree.data.grad = None
    out.backward(up, retain_graph=True)
    first = tree.data.grad
    tree.data.grad = None
    out.backward(up)
    assert _close(tree.data.grad, first)
    csrc.check_device_status()


def _query_reference(tree, pts, rows):
    with torch.no_grad():
        _, ids = tree(pts, want_node_ids=True)
    want = torch.zeros(tree.child.numel(), rows.shape[1], dtype=torch.float64, device=pts.device)
    want.index_add_(0, ids, rows.double())
    return ids, want


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8, 9, 16, 17, 28, 33, 49, 65, 76, 97, 130])
@pytest.mark.parametrize("N", [2, 3])
def test_query_rows_of_any_length(K, N, cuda_device):
    tree = svox.N3Tree(N=N, data_dim=K, data_format=None, init_refine=2, device=cuda_device)
    gen = torch.Generator(cuda_device).manual_seed(K)
    tree.data.data.normal_(generator=gen)
    flat = tree.data.data.view(-1, K)
    for Q in (1, 31, 32, 33, 1000):
        pts = torch.rand(Q, 3, generator=gen, device=cuda_device)
        rows = torch.randn(Q, K, generator=gen, device=cuda_device)
        ids, want = _query_reference(tree, pts, rows)
        tree.data.grad = None
        vals, ids2 = tree(pts, want_node_ids=True)
        assert torch.equal(ids, ids2) and torch.equal(vals, flat[ids])
        vals.backward(rows)
        got = tree.data.grad.view(-1, K)
        # a few 32-bit additions per element against double sums
        assert (got - want).abs().max().item() <= 1e-6 * max(1.0, want.abs().max().item())
        direct = csrc.query_vertical_backward(tree._spec(), pts, rows).view(-1, K)
        assert (direct - want).abs().max().item() <= 1e-6 * max(1.0, want.abs().max().item())
    csrc.check_device_status()


@pytest.mark.parametrize("K", [4, 8, 12, 28, 32, 36, 76, 128, 132, 160, 220, 224, 225])
def test_query_values_through_shared_memory(K, cuda_device):
    # records that are copied as 16-byte words, longer ones as floats, and those that go row by row;
    # into results that lie on a 16-byte boundary and beside one
    import ctypes as C
    tree = svox.N3Tree(data_dim=K, data_format=None, init_refine=2, device=cuda_device)
    gen = torch.Generator(cuda_device).manual_seed(K)
    tree.data.data.normal_(generator=gen)
    spec = tree._spec()
    for Q in (1, 5, 33, 1000):
        pts = torch.rand(Q, 3, generator=gen, device=cuda_device)
        ids, _ = _query_reference(tree, pts, torch.zeros(Q, 1, device=cuda_device))
        want = tree.data.data.view(-1, K)[ids]
        for shift in (0, 1):
            out = torch.full((Q * K + 8,), -7.0, device=cuda_device)
            t = csrc._CTree(spec.data.data_ptr(), spec.child.data_ptr(), spec.offset.data_ptr(),
                            spec.scaling.data_ptr(), tree.data.shape[0], 2, K)
            st = csrc.library().svoxb_query_vertical(
                C.byref(t), C.c_void_p(pts.data_ptr()), C.c_int64(Q),
                C.c_void_p(out.data_ptr() + 4 * shift), C.c_void_p(0),
                C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0
            assert torch.equal(out[shift:shift + Q * K].view(Q, K), want)
            assert (out[:shift] == -7).all() and (out[shift + Q * K:] == -7).all()
    csrc.check_device_status()


def test_launches_known_do_not_grow_with_the_trees(cuda_device):
    # gradients of many sizes, and logs of many numbers of bins, share a few launch configurations
    import ctypes as C
    lib = csrc.library()
    K, Q = 49, 800000
    gen = torch.Generator(cuda_device).manual_seed(3)
    rows = torch.zeros(Q, K, device=cuda_device)
    none = torch.zeros(3, device=cuda_device)
    grad = torch.empty(8 * 400000 * K, device=cuda_device)

    def backward(M):
        ids = torch.randint(0, 8 * M, (Q,), generator=gen, device=cuda_device)
        t = csrc._CTree(grad.data_ptr(), none.data_ptr(), none.data_ptr(), none.data_ptr(), M, 2, K)
        assert lib.svoxb_query_scatter(
            C.byref(t), C.c_void_p(ids.data_ptr()), C.c_int64(Q), C.c_void_p(rows.data_ptr()),
            C.c_int32(K), C.c_void_p(grad.data_ptr()), C.c_int(1),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0

    tree = _shell("SH4", 4, 2, cuda_device)
    tree.data.requires_grad_(True)
    r = svox.VolumeRenderer(tree)
    rays = _rays(20000, cuda_device)
    backward(270000)
    r(rays).sum().backward()
    before = lib.svoxb_test_known_launches()
    for M in range(270000, 390000, 4000):
        backward(M)
    try:
        for mb in range(1, 13):
            assert lib.svoxb_test_knob(5, mb) == 0
            r(rays).sum().backward()
    finally:
        lib.svoxb_test_knob(5, 32)
    # three kernels count tiles, each in at most a dozen steps; one fills bins
    assert lib.svoxb_test_known_launches() - before <= 12
    csrc.check_device_status()


@pytest.mark.parametrize("K", [97, 100])
@pytest.mark.parametrize("Q", [74000, 75000, 300001])
def test_query_backward_binned(K, Q, cuda_device):
    # 299592 slots of about 400 bytes: 116 MB and more; binned from a quarter as many points on
    tree = svox.N3Tree(data_dim=K, data_format=None, init_refine=5, device=cuda_device)
    gen = torch.Generator(cuda_device).manual_seed(Q)
    pts = torch.rand(Q, 3, generator=gen, device=cuda_device)
    rows = torch.randn(Q, K, generator=gen, device=cuda_device)
    _, want = _query_reference(tree, pts, rows)
    tree(pts).backward(rows)
    got = tree.data.grad.view(-1, K)
    assert (got - want).abs().max().item() <= 2e-6 * max(1.0, want.abs().max().item())
    csrc.check_device_status()


@pytest.mark.parametrize("K", [4, 28, 33, 49, 64, 65, 130])
@pytest.mark.parametrize("how", ["even", "dense", "hot", "ends"])
def test_query_gradient_by_tiles(K, how, cuda_device):
    # a gradient of 400 MB (or, for short rows, 800; K = 4: bins), rows summed tile by tile: tiles
    # without points, with as many as a block takes in one turn, and rows so often hit that their
    # tile is shared out among blocks; ids that are no row are left out.  (A gradient beside a 16-byte
    # boundary is added to point by point.)
    import ctypes as C
    M = -(-((400 if K > 32 else 800) << 20) // (32 * K))
    n = 8 * M
    Q = {"even": n // 3, "dense": 2 * n if K > 8 else n // 2, "hot": n // 3 + 70001, "ends": n // 3}[how]
    gen = torch.Generator(cuda_device).manual_seed(K)
    ids = torch.randint(0, n, (Q,), generator=gen, device=cuda_device)
    if how == "hot":
        ids[:70001] = 5 + 3 * (torch.arange(70001, device=cuda_device) % 3)
    elif how == "ends":
        ids = torch.where(ids % 2 == 0, torch.full_like(ids, n - 1), ids % 7)
        ids[::3] = n // 2 + ids[::3] % 2
    ids[17], ids[18] = -1, n
    rows = torch.randint(-8, 9, (Q, K), generator=gen, device=cuda_device).float()
    none = torch.zeros(3, device=cuda_device)
    ok = (ids >= 0) & (ids < n)
    want = torch.zeros(n, K, dtype=torch.float64, device=cuda_device)
    want.index_add_(0, ids[ok], rows[ok].double())
    # whole numbers whose sums stay below 2^24: exact in any order
    assert want.abs().max().item() < 1 << 24
    for shift in (0, 1):                 # 16-byte aligned gradient, and not
        grad = torch.full((n * K + shift,), float("nan"), device=cuda_device)[shift:]
        t = csrc._CTree(grad.data_ptr(), none.data_ptr(), none.data_ptr(), none.data_ptr(), M, 2, K)
        st = csrc.library().svoxb_query_scatter(
            C.byref(t), C.c_void_p(ids.data_ptr()), C.c_int64(Q), C.c_void_p(rows.data_ptr()),
            C.c_int32(K), C.c_void_p(grad.data_ptr()), C.c_int(1),
            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        assert torch.equal(grad.view(n, K).double(), want)
    csrc.check_device_status()


def _scatter(M, K, ids, rows, grad):
    import ctypes as C
    none = torch.zeros(3, device=ids.device)
    t = csrc._CTree(grad.data_ptr(), none.data_ptr(), none.data_ptr(), none.data_ptr(), M, 2, K)
    assert csrc.library().svoxb_query_scatter(
        C.byref(t), C.c_void_p(ids.data_ptr()), C.c_int64(ids.numel()),
        C.c_void_p(rows.data_ptr()), C.c_int32(K), C.c_void_p(grad.data_ptr()), C.c_int(1),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0


def _scatter_is_exact(M, K, ids, rows):
    """Rows of small whole numbers: their sums are exact in any order."""
    n = 8 * M
    want = torch.zeros(n, K, device=ids.device).index_add_(0, ids, rows)
    assert want.abs().max().item() < 1 << 24
    grad = torch.full((n, K), float("nan"), device=ids.device)
    _scatter(M, K, ids, rows, grad)
    assert torch.equal(grad, want)
    csrc.check_device_status()


@pytest.mark.parametrize("K", [33, 49, 76, 130])
@pytest.mark.parametrize("how", ["steep", "turns", "run", "end", "sparse"])
def test_query_gradient_of_clustered_points(K, how, cuda_device):
    # ranges of 4096 rows are cut into tiles where points lie densely; tiles that still have more
    # points than a block sorts at a time are written in a first turn and added to in others; a row's
    # points may fill several warps; the last range reaches beyond the buffer; few points in a tile
    M = -(-(400 << 20) // (32 * K))
    n = 8 * M
    gen = torch.Generator(cuda_device).manual_seed(K)
    base = n + n // 4 if K > 128 else n // 3
    ids = torch.randint(0, n, (base,), generator=gen, device=cuda_device)

    def near(first, rows, points):
        return first + torch.randint(0, rows, (points,), generator=gen, device=cuda_device)

    if how == "steep":
        ids = (n * 0.6 + n * 0.01 * torch.randn(base, generator=gen, device=cuda_device)).long()
    elif how == "turns":
        more = [near(20 * 4096 + 1024 * q, 1024, 3 * p) for q, p in ((1, 4000), (3, 1700))]
        ids = torch.cat([ids, *more, near(33 * 4096, 2048, 5000)])
    elif how == "run":
        ids = torch.cat([ids, near(7 * 4096 + 5, 1, 3000), near(8 * 4096 - 1, 1, 900)])
    elif how == "end":
        ids = torch.cat([ids, near(n - 300, 300, 60000)])
    else:
        # a few points in most ranges, the others (without which they would be too few to be sorted
        # at all) on one row
        few = torch.arange(n // 4096, device=cuda_device) % 70
        at = torch.repeat_interleave(torch.arange(n // 4096, device=cuda_device) * 4096, few)
        at += torch.randint(0, 4096, (at.numel(),), generator=gen, device=cuda_device)
        ids = torch.cat([at, near(n // 2, 1, base)])
    ids = ids.clamp(0, n - 1)
    lim = 2 if how == "sparse" else 9
    rows = torch.randint(1 - lim, lim, (ids.numel(), K), generator=gen, device=cuda_device).float()
    _scatter_is_exact(M, K, ids, rows)


@pytest.mark.parametrize("K", [36, 49, 64, 66, 76, 130])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_query_gradient_of_rows_at_any_address(K, offset, cuda_device):
    # rows are copied as the 16-byte words that cover them; the last row ends with its buffer
    M = -(-(400 << 20) // (32 * K))
    n = 8 * M
    gen = torch.Generator(cuda_device).manual_seed(K)
    Q = n + 5 if K > 128 else n // 3 + 5
    ids = torch.randint(0, n, (Q,), generator=gen, device=cuda_device)
    rows = torch.randint(-8, 9, (Q * K + offset,), generator=gen, device=cuda_device).float()
    _scatter_is_exact(M, K, ids, rows[offset:].view(Q, K))


@pytest.mark.parametrize("K,mb", [(24, 768), (25, 767), (25, 768), (29, 768), (30, 767), (30, 768),
                                  (33, 383), (33, 384), (128, 384), (129, 384), (129, 768)])
@pytest.mark.parametrize("more", [0, 1])
def test_query_gradient_where_the_rule_changes(K, mb, more, cuda_device):
    # bins and tiles meet at these lengths and sizes, and at one point per row
    M = -(-(mb << 20) // (32 * K))
    gen = torch.Generator(cuda_device).manual_seed(K)
    Q = 8 * M + more if K > 128 or K < 30 else 2 * M + more
    ids = torch.randint(0, 8 * M, (Q,), generator=gen, device=cuda_device)
    rows = torch.randint(-8, 9, (Q, K), generator=gen, device=cuda_device).float()
    _scatter_is_exact(M, K, ids, rows)


def _fastest(calls):
    """Shortest device time of each call, taken in turn."""
    best = [float("inf")] * len(calls)
    for _ in range(12):
        for i, call in enumerate(calls):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            call()
            b.record()
            b.synchronize()
            best[i] = min(best[i], a.elapsed_time(b))
    return best


def test_query_gradient_of_clustered_points_takes_no_longer(cuda_device):
    # (tiles cut by the average density: three times as long as for points spread evenly)
    K = 76
    M = (400 << 20) // (32 * K)
    n = 8 * M
    gen = torch.Generator(cuda_device).manual_seed(1)
    rows = torch.randn(n // 2, K, generator=gen, device=cuda_device)
    grad = torch.empty(n, K, device=cuda_device)
    even = torch.randint(0, n, (n // 2,), generator=gen, device=cuda_device)
    near = n * 0.55 + n * 0.02 * torch.randn(n // 2, generator=gen, device=cuda_device)
    near = near.long().clamp(0, n - 1)
    t_even, t_near = _fastest([lambda: _scatter(M, K, even, rows, grad),
                               lambda: _scatter(M, K, near, rows, grad)])
    assert t_near < 2 * t_even


def test_query_gradient_of_half_the_size_takes_less_time(cuda_device):
    # (with tiles of 4096 rows, too few for the device, nine tenths of it)
    K = 100
    gen = torch.Generator(cuda_device).manual_seed(1)
    calls = []
    for mb in (400, 800):
        M = (mb << 20) // (32 * K)
        Q = 4 * M
        ids = torch.randint(0, 8 * M, (Q,), generator=gen, device=cuda_device)
        rows = torch.randn(Q, K, generator=gen, device=cuda_device)
        grad = torch.empty(8 * M, K, device=cuda_device)
        calls.append(lambda M=M, ids=ids, rows=rows, grad=grad: _scatter(M, K, ids, rows, grad))
    half, whole = _fastest(calls)
    assert half < 0.8 * whole


def test_query_backward_after_the_ids_were_written_to(cuda_device):
    tree, _ = W.config1()
    tree = tree.to(cuda_device)
    pts = torch.rand(500, 3, device=cuda_device)
    vals, ids = tree(pts, want_node_ids=True)
    rows = torch.randn_like(vals)
    _, want = _query_reference(tree, pts, rows)
    ids.zero_()                                          # the points are looked up again
    tree.data.grad = None
    vals.backward(rows)
    assert (tree.data.grad.view(-1, tree.data_dim) - want).abs().max().item() <= 1e-5
    csrc.check_device_status()


def test_leaf_views_equal_indexing_by_coordinates(cuda_device):
    tree, _ = W.config1()
    tree = tree.to(cuda_device)
    aux = torch.rand(tree.child.shape, device=cuda_device)
    for key in (slice(None), slice(5, 400, 3), torch.tensor([3, 1, 2])):
        view = tree[key]
        at = tuple(k.to(cuda_device) for k in view.key)
        assert torch.equal(view.values, tree.data[at]) and torch.equal(view.aux(aux), aux[at])
    tree.data.grad = None
    (tree[:].values * 2).sum().backward()
    assert np.array_equal(tree.data.grad[tree.child == 0].unique().cpu().numpy(), [2.0])
