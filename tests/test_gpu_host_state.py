"""What the host side keeps between a forward and its backward, on a GPU: the cases in which the
kept state no longer is what the forward saw."""
import pytest
import torch
import torch.utils.checkpoint

import svox_b200 as svox
from svox_b200 import csrc
from svox_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _rays(n, dev, seed=6):
    gen = torch.Generator().manual_seed(seed)
    return svox.Rays(*[t.to(dev) for t in W.sphere_rays(n, gen, 4.0, 0.2, 0.8)])


def _tree(dev, fmt="SH4", refine=3, seed=1):
    """A filled uniform tree."""
    tree = svox.N3Tree(data_format=fmt, init_refine=refine, device=dev)
    gen = torch.Generator(dev).manual_seed(seed)
    tree.data.data.normal_(std=0.5, generator=gen)
    tree.data.data[..., -1] = 10 * torch.rand(tree.child.shape, generator=gen, device=dev)
    return tree


def _grad(tree, call, up):
    tree.data.grad = None
    call().backward(up)
    return tree.data.grad


def _close(a, b):
    # sums of the same 32-bit terms in another order: 1e-5 of the largest element, the bound that
    # the reference's own two runs of a backward keep (parity_util.assert_grad_matches_reference)
    return (a - b).abs().max().item() <= 1e-5 * b.abs().max().item()


def test_training_step_under_a_default_device(cuda_device):
    want_tree, rays = _tree(cuda_device), _rays(300, cuda_device)
    with torch.device(cuda_device):
        tree = _tree(cuda_device)
        r = svox.VolumeRenderer(tree)
        up = torch.ones(300, 3)
        got = _grad(tree, lambda: r(rays), up)
    want = _grad(want_tree, lambda: svox.VolumeRenderer(want_tree)(rays), up)
    assert got.is_cuda and _close(got, want)
    csrc.check_device_status()


def _refill(n_bytes, dev):
    """Takes up memory that was just given back and writes to it."""
    return [torch.full((n_bytes // 4,), float("nan"), device=dev) for _ in range(2)]


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("fmt", ["SH4", "RGBA"])
def test_storage_of_data_replaced_before_the_backward(fmt, fast, cuda_device):
    # neither pinned by the node nor counted as an edit; the backward takes the new storage's
    # values, as the reference does, from where they lie now
    tree = _tree(cuda_device, fmt)
    r = svox.VolumeRenderer(tree)
    rays, up = _rays(300, cuda_device), torch.ones(300, 3, device=cuda_device)
    c2w = W.look_at_cameras(1, torch.Generator().manual_seed(1), 1.6)[0].to(cuda_device)
    image_up = torch.ones(12, 16, 3, device=cuda_device)

    def image():
        return r.render_persp(c2w, width=16, height=12, fx=22.0, fast=fast)
    for call, grad_out in ((lambda: r(rays, fast=fast), up), (image, image_up)):
        for change in (lambda d: d.clone(), lambda d: d * 0.5):
            tree.data.grad = None
            out = call()
            tree.data.data = change(tree.data.data)
            held = _refill(tree.data.numel() * 4, cuda_device)
            out.backward(grad_out)
            got = tree.data.grad
            del held
            assert _close(got, _grad(tree, call, grad_out))
    csrc.check_device_status()


def test_storage_of_data_replaced_before_the_backward_of_a_query(cuda_device):
    tree = _tree(cuda_device)
    pts = torch.rand(500, 3, device=cuda_device)
    up = torch.ones(500, tree.data_dim, device=cuda_device)
    tree.data.grad = None
    out = tree(pts)
    tree.data.data = tree.data.data.clone()
    tree.child.data = tree.child.data.clone()
    held = _refill(tree.data.numel() * 4, cuda_device)
    out.backward(up)
    got = tree.data.grad
    del held
    assert _close(got, _grad(tree, lambda: tree(pts), up))
    csrc.check_device_status()


@pytest.mark.parametrize("kind", ["rays", "rays_fast", "query"])
def test_shape_of_data_changed_before_the_backward_is_refused(kind, cuda_device):
    tree = _tree(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(300, cuda_device)
    pts = torch.rand(300, 3, device=cuda_device)
    before = tree.data.data
    for other in (before[:3].clone(), torch.cat((before, before)), before.cpu()):
        out = tree(pts) if kind == "query" else r(rays, fast=kind == "rays_fast")
        tree.data.data = other
        with pytest.raises(RuntimeError):
            out.sum().backward()
        tree.data.data = before
    csrc.check_device_status()


def test_log_of_another_size_is_not_replayed(cuda_device):
    # checkpointing runs the forward again in the backward, with a log sized by what has been
    # learnt meanwhile
    tree = _tree(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(300, cuda_device)
    up = torch.ones(300, 3, device=cuda_device)
    want = _grad(tree, lambda: r(rays), up)
    old = csrc._items_per_ray
    csrc.log_estimate(wait=True)
    for first, then in ((200.0, 20.0), (20.0, 200.0)):
        tree.data.grad = None
        csrc._items_per_ray = first
        out = torch.utils.checkpoint.checkpoint(r, rays, use_reentrant=False,
                                                determinism_check="none")
        csrc.log_estimate(wait=True)
        csrc._items_per_ray = then
        out.backward(up)
        assert _close(tree.data.grad, want)
    spec, src, opt = tree._spec(), svox.render._rays_spec_from_rays(rays), r._get_options()
    out, (log, cap) = csrc.volume_render_logged(spec, src, opt)
    for bad in ((up, out.detach(), (log, cap + 1)), (up[:-1], out.detach(), (log, cap)),
                (up, out.detach()[:-1], (log, cap))):
        with pytest.raises(RuntimeError):
            csrc.volume_render_backward_replay(spec, src, opt, *bad)
        with pytest.raises(RuntimeError):
            csrc.volume_render_backward_replay_parts(spec, src, opt, *bad, 2, lambda rows: None)
    csrc._items_per_ray = old
    csrc.check_device_status()


def test_data_that_is_no_parameter(cuda_device):
    tree = _tree(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(300, cuda_device)
    up = torch.ones(300, 3, device=cuda_device)
    pts = torch.rand(200, 3, device=cuda_device)
    rows = torch.ones(200, tree.data_dim, device=cuda_device)
    want = _grad(tree, lambda: r(rays), up) * 2
    want_query = _grad(tree, lambda: tree(pts), rows) * 2
    half = (tree.data.detach() / 2).requires_grad_()
    del tree.data
    tree.data = half * 2                        # a network's output
    r(rays).backward(up, retain_graph=True)
    assert _close(half.grad, want)
    half.grad = None
    tree(pts).backward(rows)
    assert _close(half.grad, want_query)
    csrc.check_device_status()


@pytest.mark.parametrize("n", [1, 700, 40000])
def test_counts_that_size_the_log(n, cuda_device):
    tree = _tree(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(n, cuda_device)
    src, opt = svox.render._rays_spec_from_rays(rays), r._get_options()
    samples = int(csrc.march_stats(tree._spec(), src, opt)[2].sum())
    _, (log, cap) = csrc.volume_render_logged(tree._spec(), src, opt)
    warps = 24 * torch.cuda.get_device_properties(cuda_device).multi_processor_count
    assert samples <= 32 * int(log[1]) <= samples + 31 * min(warps, n)
    assert int(log[0]) <= cap
    csrc.log_estimate(wait=True)
    assert csrc._LogWatch.last_used == int(log[0]) and csrc._LogWatch.last_cap == cap


@pytest.mark.parametrize("n", [300, 12000])
def test_a_log_given_up_is_not_replayed(n, cuda_device):
    gen = torch.Generator().manual_seed(5)
    tree = W.shell_tree(4, 3, "SH9", gen, (5.0, 50.0), W._SHELL).to(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(n, cuda_device)
    up = torch.ones(n, 3, device=cuda_device)
    want = _grad(tree, lambda: r(rays), up)
    spec, src, opt = tree._spec(), svox.render._rays_spec_from_rays(rays), r._get_options()
    assert csrc.log_is_sorted(spec, n, False) == (n == 12000)
    out, (log, cap) = csrc.volume_render_logged(spec, src, opt)
    used = csrc.log_chunks_used(log)
    assert 0 < used <= cap
    log[4] = 1                                   # the mark of a forward that gave its log up
    assert csrc.log_chunks_used(log) > cap
    got = csrc.volume_render_backward_replay(spec, src, opt, up, out, (log, cap))
    assert _close(got, want)
    parts = csrc.volume_render_backward_replay_parts(spec, src, opt, up, out, (log, cap), 3,
                                                     lambda rows: None)
    assert _close(parts, want)
    # the counts that the next log is sized by are what they were
    log[4] = 0
    assert csrc.log_chunks_used(log) == used
    csrc.check_device_status()


@pytest.mark.parametrize("fmt", ["SH9", "RGBA"])
@pytest.mark.parametrize("image", [False, True])
def test_march_behind_a_log_that_was_too_small(fmt, image, cuda_device):
    # its index is built in the log's memory: no room for the table, room for the table, for some
    # of the bricks (about 4000), for all of them; and for few rays there is no index
    gen = torch.Generator().manual_seed(5)
    tree = W.shell_tree(4, 3, fmt, gen, (5.0, 50.0), W._SHELL).to(cuda_device)
    r = svox.VolumeRenderer(tree)
    spec, opt = tree._spec(), r._get_options()
    if image:
        c2w = W.look_at_cameras(1, gen, 1.6)[0].to(cuda_device)
        # 2^17 pixels (or rays) walk the tree, more build the index
        srcs = [svox.render._make_camera_spec(c2w.contiguous(), 512, h, 700.0, 700.0)
                for h in (20, 256, 257)]
    else:
        srcs = [svox.render._rays_spec_from_rays(_rays(n, cuda_device))
                for n in (5000, 1 << 17, (1 << 17) + 1)]
    old = csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS
    csrc.log_estimate(wait=True)
    try:
        for src in srcs:
            n = csrc.n_rays_of(src, image)
            for chunks in (2, 400, 3000, 20000):
                csrc.log_estimate(wait=True)
                csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS = 0.0, chunks
                out, (log, cap) = csrc.volume_render_logged(spec, src, opt, image=image)
                up = torch.linspace(-1, 1, out.numel(), device=cuda_device).view(out.shape)
                want = csrc.host().volume_render_backward(spec, src, opt, image, up, out)
                if csrc.log_chunks_used(log) <= cap:
                    continue
                for _ in range(2):               # the counters of the build are put back
                    got = csrc.volume_render_backward_replay(spec, src, opt, up, out, (log, cap),
                                                             image=image)
                    assert _close(got, want), (n, chunks)
                    got = csrc.volume_render_backward_replay_parts(
                        spec, src, opt, up, out, (log, cap), 3, lambda rows: None, image=image)
                    assert _close(got, want), (n, chunks)
    finally:
        csrc.log_estimate(wait=True)
        csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS = old
    csrc.check_device_status()


def test_march_behind_a_log_sees_softplus_densities(cuda_device):
    gen = torch.Generator().manual_seed(5)
    tree = W.shell_tree(3, 2, "SH4", gen, (5.0, 50.0), W._SHELL).to(cuda_device)
    r = svox.VolumeRenderer(tree, density_softplus=True)
    src, opt, spec = svox.render._rays_spec_from_rays(_rays(140000, cuda_device)), r._get_options(), \
        tree._spec()
    old = csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS
    csrc.log_estimate(wait=True)
    try:
        csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS = 0.0, 3000
        out, logpair = csrc.volume_render_logged(spec, src, opt)
    finally:
        csrc.log_estimate(wait=True)
        csrc._items_per_ray, csrc._LOG_SLACK_CHUNKS = old
    assert csrc.log_chunks_used(logpair[0]) > logpair[1]
    up = torch.ones_like(out)
    assert _close(csrc.volume_render_backward_replay(spec, src, opt, up, out, logpair),
                  csrc.volume_render_backward(spec, src, opt, up, out))
    csrc.check_device_status()


@pytest.mark.parametrize("n", [300, 12000])
@pytest.mark.parametrize("softplus", [False, True])
def test_diagonal_alone_equals_that_of_se_grad(n, softplus, cuda_device):
    gen = torch.Generator().manual_seed(5)
    tree = W.shell_tree(4, 3, "SH9", gen, (5.0, 50.0), W._SHELL).to(cuda_device)
    r, rays = svox.VolumeRenderer(tree, density_softplus=softplus), _rays(n, cuda_device)
    spec, src, opt = tree._spec(), svox.render._rays_spec_from_rays(rays), r._get_options()
    _, _, want = r.se_grad(rays, torch.zeros(n, 3, device=cuda_device))
    csrc.log_estimate(wait=True)
    out, (log, cap) = csrc.volume_render_logged(spec, src, opt)
    used = csrc.log_chunks_used(log)
    got = csrc.volume_render_hessdiag_replay(spec, src, opt, out, (log, cap), used)
    assert _close(got, want)
    for bad in (0, cap + 1):
        with pytest.raises(RuntimeError):
            csrc.volume_render_hessdiag_replay(spec, src, opt, out, (log, cap), bad)
    c2w = W.look_at_cameras(1, gen, 1.6)[0].to(cuda_device)
    cam = svox.render._make_camera_spec(c2w.contiguous(), 40, 30, 56.0, 56.0)
    _, _, want = r.se_grad_persp(c2w, torch.zeros(30, 40, 3, device=cuda_device), width=40,
                                 height=30, fx=56.0)
    out, (log, cap) = csrc.volume_render_logged(spec, cam, opt, image=True)
    got = csrc.volume_render_hessdiag_replay(spec, cam, opt, out, (log, cap),
                                             csrc.log_chunks_used(log), image=True)
    assert _close(got, want)
    csrc.check_device_status()


@pytest.mark.parametrize("fmt", ["RGBA", "SH1", "SH9", "SH4"])
def test_records_at_any_address(fmt, cuda_device):
    tree = _tree(cuda_device, fmt)
    r, rays = svox.VolumeRenderer(tree), _rays(300, cuda_device)
    up = torch.linspace(-1, 1, 900, device=cuda_device).view(300, 3)
    colors = torch.zeros(300, 3, device=cuda_device)
    pts = torch.rand(100, 3, device=cuda_device)
    rows = torch.ones(100, tree.data_dim, device=cuda_device)
    with torch.no_grad():
        image = r(rays)
    want, sums = _grad(tree, lambda: r(rays), up), r.se_grad(rays, colors)
    want_query = _grad(tree, lambda: tree(pts), rows)
    flat = torch.empty(tree.data.numel() + 1, device=cuda_device)
    moved = flat[1:].view(tree.data.shape)
    moved.copy_(tree.data.detach())
    tree.data = torch.nn.Parameter(moved)
    assert tree.data.data_ptr() % 16 != 0
    # other kernels: colours and gradients are each within 1e-5 of the reference's
    # (test_gpu_parity), so within 2e-5 of each other
    with torch.no_grad():
        assert (r(rays) - image).abs().max() <= 2e-5
        with r.frozen_tree():
            assert (r(rays) - image).abs().max() <= 2e-5
    assert (_grad(tree, lambda: r(rays), up) - want).abs().max() <= 2e-5 * want.abs().max()
    assert torch.equal(_grad(tree, lambda: tree(pts), rows), want_query)
    for a, b in zip(r.se_grad(rays, colors), sums):
        # (the generic march adds the density's gradient once per channel: the bound of
        # test_se_grad_through_either_log_and_without)
        assert (a - b).abs().max() <= 3e-4 * b.abs().max()
    csrc.check_device_status()


def test_forward_mode_tangents_are_refused(cuda_device):
    from torch.autograd import forward_ad
    tree = _tree(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(10, cuda_device)
    pts = torch.rand(10, 3, device=cuda_device)
    data = tree.data.detach()
    del tree.data
    with forward_ad.dual_level():
        tree.data = forward_ad.make_dual(data, torch.ones_like(data))
        for call in (lambda: r(rays), lambda: tree(pts)):
            with pytest.raises(NotImplementedError):
                call()
        tree.data = data
        assert r(rays).shape == (10, 3) and tree(pts).shape == (10, tree.data_dim)


@pytest.mark.parametrize("n", [300, 12000])
def test_training_step_in_a_graph(n, cuda_device):
    # the counts of a captured forward are nobody's: its slot would be written at every replay
    gen = torch.Generator().manual_seed(5)
    tree = W.shell_tree(4, 3, "SH9", gen, (5.0, 50.0), W._SHELL).to(cuda_device)
    r, rays = svox.VolumeRenderer(tree), _rays(n, cuda_device)
    up = torch.ones(n, 3, device=cuda_device)
    want = _grad(tree, lambda: r(rays), up).clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            _grad(tree, lambda: r(rays), up)
    torch.cuda.current_stream().wait_stream(side)
    csrc.log_estimate(wait=True)
    assert not csrc.host().logs_pending()
    tree.data.grad = None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r(rays).backward(up)
    assert not csrc.host().logs_pending()
    got = tree.data.grad
    for _ in range(2):
        got.fill_(7.0)                      # the step writes the whole gradient anew
        graph.replay()
        torch.cuda.synchronize()
        assert _close(got, want)
    before = csrc.log_estimate()
    few = svox.Rays(*[t[:10].contiguous() for t in rays])
    for _ in range(20):                     # takes every slot there is
        graph.replay()
        _grad(tree, lambda: r(few), up[:10].contiguous())
        graph.replay()
        csrc.log_estimate(wait=True)
    assert csrc.log_estimate() <= max(before, 1000.0)
    csrc.check_device_status()
