"""What the host side keeps between a forward and its backward, or from one call to the next: the
tree's edit counter, the tensors a spec is packed from, leaf views, the item log's size."""
import pytest
import torch
import torch.nn.utils.parametrize

import svox_b200 as svox
from svox_b200 import csrc

needs_build = pytest.mark.skipif(not csrc.is_built(), reason="the native library is not built")


@pytest.mark.parametrize("device", ["cpu", "meta"])
def test_edit_counter_lives_in_host_memory(device):
    # the native node reads it on the host in the backward
    with torch.device(device):
        tree = svox.N3Tree(data_format="SH1", init_refine=1, device="cpu")
    assert tree.data.device.type == "cpu"
    assert tree._data_epoch.device.type == "cpu" and tree._data_epoch.dtype == torch.int64
    before = tree._spec().data_epoch()
    tree[0, -1:] = 2.0
    assert tree._spec().data_epoch() > before


def test_edit_counter_of_a_tree_made_in_inference_mode():
    with torch.inference_mode():
        tree = svox.N3Tree(data_format="SH1")
    before = int(tree._data_epoch)
    tree._data_epoch += 1           # (an inference tensor refuses this outside that mode)
    assert int(tree._data_epoch) == before + 1


@needs_build
@pytest.mark.parametrize("counter", [torch.zeros((), dtype=torch.int64, device="meta"),
                                     torch.zeros((), dtype=torch.int32),
                                     torch.zeros(2, dtype=torch.int64)])
def test_native_node_refuses_a_counter_it_cannot_read(counter):
    tree = svox.N3Tree(data_format="SH1")
    opt = csrc.RenderOptions()
    with pytest.raises(RuntimeError, match="edit counter"):
        csrc.host().render_node(tree.data, tree._spec(), csrc.RaysSpec(), opt, False, 0, counter)


class _Doubled(torch.nn.Module):
    def forward(self, x):
        return 2 * x


def test_spec_finds_tensors_wherever_the_module_keeps_them():
    lobes = torch.rand(2, 4)
    tree = svox.N3Tree(data_format="SG2", extra_data=lobes)
    spec = tree._spec()
    assert spec.data is tree.data and spec.child is tree.child and torch.equal(spec.extra_data, lobes)
    del tree.extra_data
    tree.extra_data = torch.nn.Parameter(lobes + 1)          # lobes that are trained elsewhere
    assert tree._spec().extra_data is tree.extra_data
    tree.offset = torch.nn.Parameter(tree.offset + 1)
    assert tree._spec().offset is tree.offset
    plain = svox.N3Tree(data_format="SH1")
    assert plain._spec().extra_data is None
    plain.extra_data = lobes                                 # a plain attribute
    assert plain._spec().extra_data is lobes

    tree = svox.N3Tree(data_format="SH1")
    tree.data.data.fill_(1.5)
    torch.nn.utils.parametrize.register_parametrization(tree, "data", _Doubled())
    assert torch.equal(tree._spec().data, torch.full_like(tree.data, 3.0))

    tree = svox.N3Tree(data_format="SH1")
    made = tree.data * 2                     # what a replica, or a network that makes data, has
    del tree.data
    tree.data = made
    assert tree._spec().data is made and tree._spec(world=False).data is made

    tree = svox.N3Tree(data_format="SH1")
    other = torch.ones_like(tree.data)
    seen = []

    class Call(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.tree = tree

        def forward(self):
            seen.append(self.tree._spec().data)
    torch.func.functional_call(Call(), {"tree.data": other})
    assert seen[0] is other


class _Counts:
    """Stands in for the native module: the counts of finished forwards."""

    def __init__(self, *counts):
        self.counts = list(counts)

    def poll_logs(self):
        counts, self.counts = self.counts, []
        return counts


@pytest.mark.parametrize("samples", [2 ** 31 - 32, 2 ** 31, 2 ** 33])
def test_log_grows_for_any_number_of_samples(samples, monkeypatch):
    # 2^24 rays with up to 512 samples each, through a log of 2^31 / 8 samples
    rays, cap = 1 << 24, 1 << 23
    monkeypatch.setattr(csrc, "_items_per_ray", 8.0)
    monkeypatch.setattr(csrc, "host", lambda: _Counts((samples // 32, samples // 32, rays, cap)))
    need = samples // 32
    assert need <= csrc.log_capacity(rays) <= 1.25 * need + csrc._LOG_SLACK_CHUNKS + 1


def test_a_log_given_up_does_not_size_the_next_one(monkeypatch):
    # the head of such a log holds the chunks that were really asked for; the mark is a word of
    # its own, which the host does not look at
    monkeypatch.setattr(csrc, "_items_per_ray", 8.0)
    monkeypatch.setattr(csrc, "host", lambda: _Counts((2000, 1500, 1000, 40000)))
    assert csrc.log_capacity(1000) <= 2000 + csrc._LOG_SLACK_CHUNKS


_DRIVER = r"""
#include "open_groups.h"
using namespace svoxb;
// Looks in the entry that group `other` published for each of the groups lo .. hi - 1 that share
// its place: how many take it for theirs without being `other`, or the other way round.
extern "C" int mistaken(uint32_t lo, uint32_t hi, uint32_t other, int id) {
    const uint64_t entry = open_group_entry(other, id);
    int n_wrong = open_group_id(entry) != id;
    for (uint32_t n = lo; n < hi; ++n)
        if (open_group_place(n) == open_group_place(other))
            n_wrong += open_group_is(entry, n) != (n == other) || open_group_is(0, n);
    return n_wrong;
}
"""


def test_open_groups_are_never_mistaken(tmp_path):
    # whatever the group is that a late reader finds, or a late writer overwrites
    import ctypes
    import os
    import subprocess
    src, lib = tmp_path / "driver.cpp", tmp_path / "driver.so"
    src.write_text(_DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                    os.path.dirname(csrc.__file__), str(src), "-o", str(lib)], check=True)
    mistaken = ctypes.CDLL(str(lib)).mistaken
    for other in (0, 7, 8, 255, 256, 511, 4096, (1 << 25) - 1):
        for id_ in (0, 0xffffff, 0x7fffffff):
            assert mistaken(max(0, other - 5000), other + 5000, other, id_) == 0


def test_se_grad_repeats_with_a_larger_log_and_marches_at_last(monkeypatch):
    calls = []
    tree = csrc.TreeSpec()
    tree._weight_accum = torch.zeros(8)

    class Module:
        def __init__(self, used):
            self.used = list(used)

        def poll_logs(self):
            return []

        def se_grad(self, tree, src, opt, image, colors, cap, checked, watch):
            calls.append((cap, checked, watch, tree._weight_accum))
            return "out", "grad", "hess", self.used.pop(0)
    rays = csrc.RaysSpec()
    for n, checked in ((4096, False), (4097, True)):
        rays.origins = torch.zeros(n, 3)
        calls.clear()
        module = Module([0])
        monkeypatch.setattr(csrc, "host", lambda: module)
        assert csrc.se_grad(tree, rays, None, None) == ("out", "grad", "hess")
        assert [c[1:3] for c in calls] == [(checked, True)]
    calls.clear()
    module = Module([10 ** 6, 10 ** 6 - 1])
    assert csrc.se_grad(tree, rays, None, None) == ("out", "grad", "hess")
    assert calls[0][0] < 10 ** 6 < calls[1][0] and [c[2] for c in calls] == [True, False]
    # weights are accumulated once
    assert calls[0][3] is tree._weight_accum is not None and calls[1][3] is None
    calls.clear()
    module = Module([2 ** 63 - 1] * 4)               # given up every time
    out = torch.ones(n, 3)
    monkeypatch.setattr(Module, "se_grad", lambda self, *a: (out, None, None, self.used.pop(0)))
    seen = []
    monkeypatch.setattr(csrc, "se_grad_march",
                        lambda *a, **k: seen.append((a[3], a[4].shape)) or ("g", "h"))
    got = csrc.se_grad(tree, rays, None, torch.zeros(3 * n))
    assert got[0] is out and got[1:] == ("g", "h") and seen == [(out, out.shape)]


def test_aux_of_a_view_made_before_a_refine():
    tree = svox.N3Tree(data_format="SH1", init_refine=1)
    view, aux = tree[:], torch.rand(tree.child.shape)
    want = aux[view.key]
    assert torch.equal(view.aux(aux), want)
    tree.refine(sel=(torch.tensor([3]), torch.tensor([0]), torch.tensor([1]), torch.tensor([0])))
    assert torch.equal(view.aux(aux), want)              # the leaves it was made of
    grown = torch.cat((aux, torch.rand(5, 2, 2, 2)))
    assert torch.equal(view.aux(grown), want)
    with pytest.raises(RuntimeError):
        view.values
    view = tree[:]
    larger = torch.rand(tree.child.shape[0], 3, 3, 3)    # not of the tree's branching
    assert torch.equal(view.aux(larger), larger[view.key])
    assert (view.aux(larger.numpy()) == larger[view.key].numpy()).all()
    with pytest.raises(IndexError):
        view.aux(torch.rand(100))


@pytest.mark.parametrize("fmt,floats", [("RGBA", 4), ("SH1", 4), ("SH9", 28), ("SH4", 13)])
def test_records_that_cannot_be_read_in_words_are_not_logged(fmt, floats):
    # they are rendered and differentiated by the kernels for any alignment
    opt = csrc.RenderOptions()
    opt.format = csrc.FORMAT_RGBA if fmt == "RGBA" else csrc.FORMAT_SH
    opt.basis_dim = (floats - 1) // 3 if fmt != "RGBA" else -1
    tree = csrc.TreeSpec()
    flat = torch.zeros(8 * floats + 4)
    for shift in range(4):
        tree.data = flat[shift:shift + 8 * floats].view(1, 2, 2, 2, floats)
        whole = tree.data.data_ptr() % 16 == 0
        assert csrc.log_eligible(tree, opt) == (whole or floats % 4 != 0)
    tree.data = torch.empty(1 << 28, 2, 2, 2, floats, device="meta")
    assert not csrc.log_eligible(tree, opt)              # more nodes than the log has bits for


def test_forward_mode_tangents_are_refused():
    from torch.autograd import forward_ad
    from svox_b200.tree import _QueryVerticalFunction
    data = torch.zeros(1, 2, 2, 2, 4)
    csrc.refuse_tangent(data)
    with forward_ad.dual_level():
        csrc.refuse_tangent(data)
        dual = forward_ad.make_dual(data, torch.ones_like(data))
        with pytest.raises(NotImplementedError):
            csrc.refuse_tangent(dual)
        with pytest.raises(NotImplementedError):
            _QueryVerticalFunction.apply(dual, None, torch.zeros(1, 3))
    csrc.refuse_tangent(data)
