"""What the host side keeps between a forward and its backward, on a GPU: the cases in which the
kept state no longer is what the forward saw."""
import pytest
import torch

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
