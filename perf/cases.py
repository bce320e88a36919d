"""Workloads by which this package's speed is judged: point queries, ray batches, images, weight
accumulation and Gauss-Newton gradients, each through the public API.

The scenes are the synthetic ones of ``svox_b200.workloads`` (a uniform tree, one spherical shell
refined three more levels, three overlapping shells), built and filled on the GPU from a seed.
"""
import functools
import math

import numpy as np
import torch

import svox_b200 as svox

DEVICE = "cuda"

# (centre, inner radius, outer radius) of the occupied shells
SHELLS = {
    "uniform": (),
    "shell": (((0.5, 0.5, 0.5), 0.30, 0.35),),
    "shells": (((0.42, 0.55, 0.47), 0.185, 0.215), ((0.60, 0.38, 0.52), 0.235, 0.265),
               ((0.50, 0.50, 0.62), 0.135, 0.165)),
}


def _case(name, kind, tree, refine, extra, fmt, **more):
    case = {"kind": kind, "tree": tree, "refine": refine, "extra": extra, "format": fmt,
            "n": 0, "width": 0, "height": 0, "views": 0, "grad": False, "fast": False,
            "frozen": False, "softplus": False, "op": ""}
    case.update(more)
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # a handful of look-ups in a toy scene: interactive probing, unit-test sized programs
        _case("query_tiny", "query", "uniform", 3, 0, "SH4", n=1000),
        # supervising leaf values directly at sampled points, one optimisation step
        _case("query_step", "query", "uniform", 6, 0, "SH9", n=200003, grad=True),
        # the 2^24-point query of the benchmark, values and gradient
        _case("query_full_step", "query", "uniform", 7, 0, "SH16", n=1 << 24, grad=True),
        # the toy training step: 4096 leaves, 4096 rays
        _case("rays_toy_step", "rays", "uniform", 3, 0, "SH4", n=4096, grad=True),
        # one stochastic step on a 512^3 scene with the ray batch of a NeRF-style trainer
        _case("rays_batch_step", "rays", "shell", 5, 3, "SH9", n=4096, grad=True),
        # the benchmark's training step: 2^20 rays
        _case("rays_full_step", "rays", "shell", 5, 3, "SH9", n=1 << 20, grad=True),
        # one evaluation view of a 512^3 scene
        _case("image_view", "image", "shell", 5, 3, "SH16", width=800, height=800, views=1),
        # optimising a tree image by image
        _case("image_step", "image", "shell", 5, 3, "SH16", width=800, height=800, views=1,
              grad=True),
        # a viewer orbiting a 1024^3 scene that does not change, with the early-stop thresholds
        _case("image_orbit", "image", "shells", 6, 3, "SH16", width=1920, height=1080, views=4,
              fast=True, frozen=True),
        # the default record format (plain colours), one training step of a ray batch
        _case("rgba_step", "rays", "shell", 4, 3, "RGBA", n=65536, grad=True),
        # which leaves are seen at all: the pruning pass after extraction
        _case("weights_max", "weights", "shell", 5, 3, "SH9", width=800, height=800, views=2,
              op="max"),
        # gradient and Gauss-Newton diagonal of a ray batch, for second-order optimisers
        _case("se_grad_rays", "se_grad", "shell", 5, 3, "SH9", n=100000),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]; every other one is odd."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.5 else n))


def _scene(rng):
    if rng.random() < 0.3:
        return "uniform", rng.choice((3, 4, 5, 6)), 0
    return "shell", rng.choice((4, 5)), rng.choice((2, 3))


def _dims(fmt):
    """(record length, basis functions per channel) of a format."""
    if fmt == "RGBA":
        return 4, 1
    b = int("".join(c for c in fmt if c.isdigit()))
    return 3 * b + 1, b


def draw(rng):
    kind = rng.choice(("query", "query", "rays", "rays", "rays", "image", "image", "weights",
                       "se_grad"))
    tree, refine, extra = _scene(rng)
    if kind == "query":
        fmt = rng.choice(("RGBA", "SH1", "SH4", "SH9", "SH16"))
        return _case(None, kind, tree, refine, extra, fmt,
                     n=_log_int(rng, 1, 1 << 22), grad=rng.random() < 0.5)
    fmt = rng.choice(("RGBA", "SH4", "SH9", "SH9", "SH16", "SH25", "SG9"))
    k, _ = _dims(fmt)
    if kind == "rays":
        softplus = rng.random() < 0.1
        most = (1 << 20) * 28 // max(k, 28) // (8 if softplus or fmt in ("RGBA", "SG9") else 2)
        return _case(None, kind, tree, refine, extra, fmt, n=_log_int(rng, 1, most),
                     grad=rng.random() < 0.6, softplus=softplus)
    if kind == "image":
        grad = rng.random() < 0.4
        width = _log_int(rng, 32, 640 if fmt in ("RGBA", "SH25", "SG9") else 1000)
        return _case(None, kind, tree, refine, extra, fmt, width=width,
                     height=max(16, width * rng.choice((9, 10, 12, 16)) // 16),
                     views=1 if grad else rng.choice((1, 1, 3)), grad=grad,
                     fast=not grad and rng.random() < 0.4,
                     frozen=not grad and rng.random() < 0.3)
    if kind == "weights":
        width = _log_int(rng, 64, 640)
        return _case(None, kind, tree, refine, extra, rng.choice(("RGBA", "SH4", "SH9", "SH16")),
                     width=width, height=width, views=rng.choice((1, 2)),
                     op=rng.choice(("sum", "max")))
    return _case(None, kind, tree, refine, extra, rng.choice(("RGBA", "SH4", "SH9", "SH16")),
                 n=_log_int(rng, 100, 100000))


# ---------------------------------------------------------------------------
# Scenes, rays and cameras

def _in_shells(centers, shells):
    inside = torch.zeros(centers.shape[0], dtype=torch.bool, device=centers.device)
    for c, lo, hi in shells:
        dist = (centers - torch.tensor(c, device=centers.device)).norm(dim=1)
        inside |= (dist >= lo) & (dist <= hi)
    return inside


def _offsets(device):
    cell = torch.arange(8, device=device)
    return torch.stack(((cell >> 2) & 1, (cell >> 1) & 1, cell & 1), dim=1).float()


def _node_corners(tree):
    """Lower corner of every node, level by level down from the root."""
    slot, depth = tree.parent_depth[:, 0].long(), tree.parent_depth[:, 1]
    corner = torch.zeros(slot.shape[0], 3, device=slot.device)
    offset = _offsets(slot.device)
    for d in range(1, int(depth.max()) + 1):
        at = torch.nonzero(depth == d).flatten()
        corner[at] = corner[slot[at] // 8] + offset[slot[at] % 8] * 0.5 ** d
    return corner, depth


def _build_tree(case, gen):
    fmt, shells = case["format"], SHELLS[case["tree"]]
    more = {}
    if fmt.startswith("SG"):
        lobes = _dims(fmt)[1]
        axis = torch.randn(lobes, 3, generator=gen, device=DEVICE)
        sharp = torch.rand(lobes, 1, generator=gen, device=DEVICE) * 4 + 1
        more["extra_data"] = torch.cat((sharp, axis / axis.norm(dim=1, keepdim=True)), dim=1)
    tree = svox.N3Tree(N=2, data_format=fmt, init_refine=case["refine"], device=DEVICE, **more)
    if shells:
        view = tree[:]
        centers = view.corners_local + 0.5 * view.lengths_local[:, None]
        tree[_in_shells(centers, shells).cpu()].refine(case["extra"])
    with torch.no_grad():
        data = tree.data.data
        if case["kind"] == "query":
            data.normal_(generator=gen)
            return tree
        data.normal_(std=0.5, generator=gen)
        sigma = torch.rand(data.shape[:-1], generator=gen, device=DEVICE)
        empty = -12.0 if case["softplus"] else 0.0
        if not shells:
            data[..., -1] = 10.0 * sigma
        else:
            corner, depth = _node_corners(tree)
            half = 0.5 ** (depth.float() + 2)
            centers = corner[:, None] + half[:, None, None] * (2 * _offsets(DEVICE) + 1)
            inside = _in_shells(centers.reshape(-1, 3), shells).view(sigma.shape)
            inside &= (depth == case["refine"] + case["extra"])[:, None, None, None]
            data[..., -1] = torch.where(inside, 5.0 + 45.0 * sigma, empty)
    return tree


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _rays(n, gen):
    """Rays from a sphere around the scene towards points inside it."""
    origins = 0.5 + 4.0 * _unit(torch.randn(n, 3, generator=gen, device=DEVICE))
    targets = 0.2 + 0.6 * torch.rand(n, 3, generator=gen, device=DEVICE)
    dirs = _unit(targets - origins)
    return svox.Rays(origins=origins, dirs=dirs, viewdirs=dirs.clone())


def _cameras(n, gen):
    """Camera-to-world matrices on a sphere, looking at the centre of the scene, from where the
    scene's cube about fills the frame."""
    back = _unit(torch.randn(n, 3, generator=gen, device=DEVICE))
    up = torch.tensor([0.0, 0.0, 1.0], device=DEVICE).expand(n, 3)
    right = _unit(torch.linalg.cross(-back, up))
    return torch.stack((right, torch.linalg.cross(right, -back), back, 0.5 + 1.6 * back), dim=2)


class _State:
    pass


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    s = _State()
    s.case = case
    s.tree = _build_tree(case, gen)
    s.tree.data.requires_grad_(case["grad"])
    shape = (case["height"], case["width"])
    if case["kind"] == "query":
        s.points = torch.rand(case["n"], 3, generator=gen, device=DEVICE)
        shape = (case["n"], s.tree.data_dim)
    else:
        s.renderer = svox.VolumeRenderer(s.tree, density_softplus=case["softplus"])
        shape = (*shape, 3)
        if case["n"]:
            s.rays = _rays(case["n"], gen)
            shape = (case["n"], 3)
        else:
            s.cameras = list(_cameras(case["views"], gen))
            s.focal = 1.4 * case["width"]
    if case["grad"]:        # gradient of the user's loss with respect to the call's result
        s.upstream = torch.randn(shape, generator=gen, device=DEVICE)
    if case["kind"] == "se_grad":
        s.colors = torch.rand(shape, generator=gen, device=DEVICE)
    return s


# ---------------------------------------------------------------------------
# One pass

def _view(s, c2w):
    case = s.case
    return s.renderer.render_persp(c2w, width=case["width"], height=case["height"], fx=s.focal,
                                   fast=case["fast"])


def run(s):
    case, tree = s.case, s.tree
    kind = case["kind"]
    if kind == "se_grad":
        return s.renderer.se_grad(s.rays, s.colors)
    if kind == "weights":
        with torch.no_grad(), tree.accumulate_weights(op=case["op"]) as accum:
            images = [_view(s, c2w) for c2w in s.cameras]
        return images, accum()
    if case["grad"]:
        tree.data.grad = None
        if kind == "query":
            out, ids = tree(s.points, want_node_ids=True)
        else:
            out, ids = s.renderer(s.rays) if kind == "rays" else _view(s, s.cameras[0]), None
        out.backward(s.upstream)
        return {"out": out.detach(), "ids": ids, "grad": tree.data.grad}
    with torch.no_grad():
        if kind == "query":
            return tree(s.points, want_node_ids=True)
        if kind == "rays":
            return s.renderer(s.rays)
        if case["frozen"]:
            with s.renderer.frozen_tree():
                return [_view(s, c2w) for c2w in s.cameras]
        return [_view(s, c2w) for c2w in s.cameras]


# ---------------------------------------------------------------------------
# What a pass cannot do without

@functools.lru_cache(maxsize=None)
def _scene_size(tree, refine, extra):
    """(nodes, occupied leaves) of a scene."""
    nodes = sum(8 ** level for level in range(refine + 1))
    side = 2 << refine
    if not SHELLS[tree]:
        return nodes, side ** 3
    axis = (np.arange(side) + 0.5) / side
    inside = np.zeros((side, side, side), dtype=bool)
    volume = 0.0
    for c, lo, hi in SHELLS[tree]:
        d = [(axis - c[a]) ** 2 for a in range(3)]
        r2 = d[0][:, None, None] + d[1][None, :, None] + d[2][None, None, :]
        inside |= (r2 >= lo * lo) & (r2 <= hi * hi)
        volume += 4.0 / 3.0 * math.pi * (hi ** 3 - lo ** 3)
    split = int(inside.sum())
    nodes += split * sum(8 ** level for level in range(extra))
    return nodes, int(min(0.9 * split * 8 ** extra, volume * (side << extra) ** 3))


def work(case):
    k, basis = _dims(case["format"])
    nodes, occupied = _scene_size(case["tree"], case["refine"], case["extra"])
    slots = nodes * 8
    n = case["n"]
    if case["kind"] == "query":
        touched = min(slots, n)
        bytes_ = n * (12 + 4 * k + 8) + touched * (4 + 4 * k)
        if case["grad"]:
            bytes_ += n * (12 + 4 * k) + slots * 4 * k
        return {"bytes": bytes_, "flops": n * (30 + (k if case["grad"] else 0))}
    side = (2 << case["refine"]) << case["extra"]
    rays = n or case["width"] * case["height"] * case["views"]
    # samples per ray: leaves crossed, and those of them that hold something
    visits = 1.2 * side if case["tree"] == "uniform" else (0.31 if n else 0.19) * side
    filled = (0.13 if n else 0.05) * side
    if case["tree"] == "uniform" or case["softplus"]:
        filled = visits
    if case["fast"]:
        visits, filled = 0.6 * visits, 0.5 * filled
    touched = min(slots if case["softplus"] else occupied, rays * filled)
    bytes_ = rays * ((36 if n else 0) + 12)
    bytes_ += touched * 4 * k + min(slots, rays * visits) * 4
    flops = rays * (visits * 60 + filled * (6 * basis + 60))
    if case["grad"]:
        bytes_ += rays * 12 + slots * 4 * k
        flops += rays * filled * (6 * basis + 40)
    if case["kind"] == "se_grad":
        bytes_ += rays * 12 + 2 * slots * 4 * k
        flops += rays * filled * (12 * basis + 60)
    if case["kind"] == "weights":
        bytes_ += 2 * slots * 4
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["kind"] == "query" and not case["grad"]:
        return "exact"
    # 32-bit sums of up to some hundred terms whose order is free; a gradient element is a
    # difference of sums that nearly cancel, and most of a scene's elements are zero, so a
    # single element may be off by more of the root mean square
    grad = case["grad"] or case["kind"] == "se_grad"
    return {"rel": 1e-5, "max": 2e-3 if grad else 1e-4}
