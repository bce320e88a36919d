"""Host-side mirror of the reference's native module ``svox.csrc``.

Same spec classes (``TreeSpec``, ``RaysSpec``, ``CameraSpec``,
``RenderOptions``) and the same functions with the same arguments and
results as the reference's pybind11 module (svox/csrc/svox.cpp:63-122), but
implemented by the C-ABI library ``libsvox_b200.so`` (hand-written sm_100a
kernels) loaded with ctypes; the hot calls go through the extension ``_host``.
Tensors are allocated by PyTorch and handed to the library as raw device
pointers together with the current CUDA stream.

There is no CPU implementation: if the library is missing or a tensor is
not on a CUDA device, the call raises.
"""
import copy
import ctypes as C
import os

import torch
from torch.autograd import forward_ad as _fwd

_HERE = os.path.dirname(os.path.abspath(__file__))
# SVOXB_LIBRARY: load another build of the library (e.g. one compiled with other flags)
LIB_PATH = os.environ.get("SVOXB_LIBRARY") or os.path.join(_HERE, "libsvox_b200.so")

FORMAT_RGBA, FORMAT_SH, FORMAT_SG, FORMAT_ASG = 0, 1, 2, 3
ERR_TOO_LARGE = 8   # svoxb status: a size limit


class _CTree(C.Structure):
    _fields_ = [("data", C.c_void_p), ("child", C.c_void_p), ("offset", C.c_void_p),
                ("scaling", C.c_void_p), ("M", C.c_int64), ("N", C.c_int32), ("K", C.c_int32),
                ("weight_accum", C.c_void_p), ("weight_accum_max", C.c_int32),
                ("reserved_", C.c_int32), ("extra_data", C.c_void_p),
                ("extra_rows", C.c_int32), ("extra_cols", C.c_int32)]


class _CRays(C.Structure):
    _fields_ = [("origins", C.c_void_p), ("dirs", C.c_void_p), ("vdirs", C.c_void_p),
                ("Q", C.c_int64)]


class _CCamera(C.Structure):
    _fields_ = [("c2w", C.c_void_p), ("fx", C.c_float), ("fy", C.c_float),
                ("width", C.c_int32), ("height", C.c_int32)]


class _COptions(C.Structure):
    _fields_ = [("step_size", C.c_float), ("background_brightness", C.c_float),
                ("format", C.c_int32), ("basis_dim", C.c_int32), ("ndc_width", C.c_int32),
                ("ndc_height", C.c_int32), ("ndc_focal", C.c_float), ("min_comp", C.c_int32),
                ("max_comp", C.c_int32), ("sigma_thresh", C.c_float),
                ("stop_thresh", C.c_float), ("density_softplus", C.c_int32),
                ("rgb_padding", C.c_float)]


# ---------------------------------------------------------------------------
# Spec objects: plain attribute bags with the reference's field names.

class TreeSpec:
    def __init__(self):
        self.data = self.child = self.parent_depth = self.extra_data = None
        self.offset = self.scaling = None
        self._weight_accum = None
        self._weight_accum_max = False
        self._owner = None          # weak reference to the N3Tree this spec was packed from

    def data_epoch(self):
        """Counter of the owning tree's in-place edits of ``data`` that autograd's version
        counter does not see (``tree[...] = v`` writes through ``data.data``); -1 without
        an owner."""
        tree = self._owner() if self._owner is not None else None
        return int(tree._data_epoch) if tree is not None else -1


class RaysSpec:
    def __init__(self):
        self.origins = self.dirs = self.vdirs = None


class CameraSpec:
    def __init__(self):
        self.c2w = None
        self.fx = self.fy = 0.0
        self.width = self.height = 0


class RenderOptions:
    def __init__(self):
        self.step_size = 1e-3
        self.background_brightness = 1.0
        self.format = FORMAT_RGBA
        self.basis_dim = -1
        self.ndc_width = -1
        self.ndc_height = -1
        self.ndc_focal = 0.0
        self.min_comp = 0
        self.max_comp = 0
        self.sigma_thresh = 0.0
        self.stop_thresh = 0.0
        self.density_softplus = False
        self.rgb_padding = 0.0

    def _pack(self):
        return _COptions(self.step_size, self.background_brightness, int(self.format),
                         int(self.basis_dim), int(self.ndc_width), int(self.ndc_height),
                         float(self.ndc_focal), int(self.min_comp), int(self.max_comp),
                         self.sigma_thresh, self.stop_thresh, int(bool(self.density_softplus)),
                         self.rgb_padding)


# ---------------------------------------------------------------------------
_lib = None


def library():
    """The loaded C-ABI library; raises if it has not been built."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(
                f"svox_b200: native library {LIB_PATH} not found; build it with "
                "`python -m svox_b200.csrc.build` (needs nvcc). There is no CPU fallback.")
        lib = C.CDLL(LIB_PATH)
        for name in ("svoxb_strerror", "svoxb_last_cuda_error", "svoxb_version"):
            getattr(lib, name).restype = C.c_char_p
        _lib = lib
    return _lib


_extension = None


def host():
    """The Python extension that makes the hot calls (host.cpp), bound to ``library()``."""
    global _extension
    if _extension is None:
        library()
        try:
            from . import _host as module
        except ImportError as e:
            raise RuntimeError(
                "svox_b200: the host extension is missing or does not load; build it with "
                f"`python -m svox_b200.csrc.build` ({e})") from e
        module.load(LIB_PATH)
        _extension = module
    return _extension


def is_built():
    return os.path.exists(LIB_PATH) and os.path.exists(os.path.join(_HERE, "_host.so"))


def _raise(status, what):
    lib = library()
    msg = lib.svoxb_strerror(int(status)).decode()
    cuda = lib.svoxb_last_cuda_error().decode()
    raise RuntimeError(f"svox_b200.{what}: {msg}" + (f" ({cuda})" if cuda else ""))


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


# Optional per-call device timing (used by the benchmark): when a list is
# installed with ``set_timing``, every library call appends
# (name, start_event, end_event), recorded on the launching stream around the
# call's kernels only (output zero-fill excluded).
_timing = None


def set_timing(records):
    global _timing
    _timing = records


class _timed:
    def __init__(self, name):
        self.name = name

    def __enter__(self):
        if _timing is not None:
            self.a = torch.cuda.Event(enable_timing=True)
            self.b = torch.cuda.Event(enable_timing=True)
            self.a.record()

    def __exit__(self, *exc):
        if _timing is not None:
            self.b.record()
            _timing.append((self.name, self.a, self.b))


def _check_input(x, name, dtype=torch.float32):
    # mirrors CHECK_INPUT (svox/csrc/include/data_spec.hpp:37-42) plus the dtype
    # check the reference leaves out
    if not torch.is_tensor(x):
        raise RuntimeError(f"{name} must be a tensor")
    if not x.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor")
    if not x.is_contiguous():
        raise RuntimeError(f"{name} must be contiguous")
    if x.dtype != dtype:
        raise RuntimeError(f"{name} must be {dtype} (this build computes in float32 only)")


def _pack_tree(tree):
    for n in ("data", "offset", "scaling"):
        _check_input(getattr(tree, n), n)
    _check_input(tree.child, "child", torch.int32)
    d = tree.data
    if d.dim() != 5 or tree.child.dim() != 4 or tuple(tree.child.shape) != tuple(d.shape[:4]):
        raise RuntimeError("data must be (M,N,N,N,K) and child (M,N,N,N)")
    dev = d.device
    for n in ("child", "offset", "scaling"):
        if getattr(tree, n).device != dev:
            raise RuntimeError(f"{n} must be on the same device as data")
    wa = tree._weight_accum
    wa_ptr = 0
    if wa is not None and wa.numel():
        _check_input(wa, "_weight_accum")
        if tuple(wa.shape) != tuple(tree.child.shape) or wa.device != dev:
            raise RuntimeError("_weight_accum must have the shape and device of child")
        wa_ptr = wa.data_ptr()
    ex = tree.extra_data
    ex_ptr = ex_rows = ex_cols = 0
    if ex is not None and ex.numel():
        _check_input(ex, "extra_data")
        if ex.dim() != 2 or ex.device != dev:
            raise RuntimeError("extra_data must be (basis_dim, C) on the device of data")
        ex_ptr, (ex_rows, ex_cols) = ex.data_ptr(), ex.shape
    return _CTree(d.data_ptr(), tree.child.data_ptr(), tree.offset.data_ptr(),
                  tree.scaling.data_ptr(), d.shape[0], d.shape[1], d.shape[4], wa_ptr,
                  1 if tree._weight_accum_max else 0, 0, ex_ptr, ex_rows, ex_cols)


def _pack_rays(rays, dev):
    for n in ("origins", "dirs", "vdirs"):
        t = getattr(rays, n)
        _check_input(t, n)
        if t.dim() != 2 or t.shape[1] != 3:
            raise RuntimeError(f"{n} must be (Q, 3)")
        if t.device != dev:
            raise RuntimeError(f"{n} must be on the same device as the tree")
    Q = rays.origins.shape[0]
    if rays.dirs.shape[0] != Q or rays.vdirs.shape[0] != Q:
        raise RuntimeError("origins, dirs and vdirs must have the same length")
    return _CRays(rays.origins.data_ptr(), rays.dirs.data_ptr(), rays.vdirs.data_ptr(), Q)


def _pack_camera(cam, dev):
    _check_input(cam.c2w, "c2w")
    if cam.c2w.dim() != 2 or cam.c2w.shape[1] != 4 or cam.c2w.shape[0] not in (3, 4):
        raise RuntimeError("c2w must be (3, 4) or (4, 4)")
    if cam.c2w.device != dev:
        raise RuntimeError("c2w must be on the same device as the tree")
    return _CCamera(cam.c2w.data_ptr(), float(cam.fx), float(cam.fy), int(cam.width),
                    int(cam.height))


def _out_dim(opt, K):
    # get_out_data_dim, svox/csrc/rt_kernel.cu:1009-1015
    return (K - 1) // opt.basis_dim if opt.format != FORMAT_RGBA else K - 1


def _check_indices(indices):
    _check_input(indices, "indices")
    if indices.dim() != 2 or indices.shape[1] != 3:
        raise RuntimeError("indices must be (Q, 3)")


# ---------------------------------------------------------------------------
# Functions of the reference module

def query_vertical(tree, indices):
    """-> (values (Q, K) float32, node_ids (Q,) int64); svox_kernel.cu:120-143."""
    return host().query_vertical(tree, indices)


_side_streams = {}


def zero_beside(buf):
    """Clear ``buf`` on a side stream of its device, after the work already queued on the
    current stream (the memory's previous users); -> the event after which it is zero.  The
    fill then runs beside whatever the current stream does next."""
    dev = buf.device
    side = _side_streams.get(dev)
    if side is None:
        side = _side_streams[dev] = torch.cuda.Stream(device=dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):
        buf.zero_()
        done = torch.cuda.Event()
        done.record(side)
    # should the tensor be dropped before anyone waited for the fill: its memory must not be
    # handed out again while the side stream still writes to it
    if buf.untyped_storage().size() and not _is_symmetric(buf):
        buf.record_stream(side)
    return done


def _is_symmetric(buf):
    """Symmetric-memory allocations do not come from the caching allocator."""
    try:
        from ..distributed import MulticastGradient
    except ImportError:         # torch.distributed not built
        return False
    mc = MulticastGradient.active
    return mc is not None and mc.owns(buf)


def query_vertical_backward(tree, indices, grad_output, zeroed=None):
    """-> gradient w.r.t. data, (M, N, N, N, Kg); svox_kernel.cu:160-182.  ``zeroed``: a zero
    tensor of that shape to add the rows into (else one is made and cleared here)."""
    return host().query_vertical_backward(tree, indices, grad_output, zeroed)


def assign_vertical(tree, indices, values):
    """Write row q of ``values`` (Q, Kv <= K) into the record of the leaf that holds point q
    (in place, into ``tree.data``); svox_kernel.cu:80-89,145-158."""
    lib = library()
    ct = _pack_tree(tree)
    _check_indices(indices)
    _check_input(values, "values")
    Q = indices.shape[0]
    if values.dim() != 2 or values.shape[0] != Q or not 1 <= values.shape[1] <= ct.K:
        raise RuntimeError("values must be (Q, Kv) with 1 <= Kv <= K")
    with torch.cuda.device(indices.device):
        st = lib.svoxb_assign_vertical(
            C.byref(ct), C.c_void_p(indices.data_ptr()), C.c_int64(Q),
            C.c_void_p(values.data_ptr()), C.c_int32(values.shape[1]),
            C.c_void_p(tree.data.data_ptr()), _stream())
    if st:
        _raise(st, "assign_vertical")


def calc_corners(tree, indexer):
    """Lower corners (Q, 3), tree-local, of the cells ``indexer`` (Q, 4) int64 =
    (node, i, j, k); svox_kernel.cu:91-115,184-203."""
    lib = library()
    ct = _pack_tree(tree)
    _check_input(indexer, "indexer", torch.int64)
    _check_input(tree.parent_depth, "parent_depth", torch.int32)
    if indexer.dim() != 2 or indexer.shape[1] != 4:
        raise RuntimeError("indexer must be (Q, 4)")
    if tuple(tree.parent_depth.shape) != (ct.M, 2) or tree.parent_depth.device != indexer.device:
        raise RuntimeError("parent_depth must be (M, 2) on the device of indexer")
    Q = indexer.shape[0]
    with torch.cuda.device(indexer.device):
        out = torch.empty((Q, 3), dtype=tree.data.dtype, device=indexer.device)
        st = lib.svoxb_calc_corners(
            C.byref(ct), C.c_void_p(tree.parent_depth.data_ptr()),
            C.c_void_p(indexer.data_ptr()), C.c_int64(Q), C.c_void_p(out.data_ptr()),
            _stream())
    if st:
        _raise(st, "calc_corners")
    return out


def render_scratch(tree, opt):
    """The forward render's index of the tree (a table of its upper levels and bricks below it, 8
    bytes per cell) as an int32 tensor, for ``volume_render[_image](..., prepared=...)``: valid until
    the tree, ``opt.sigma_thresh`` or ``opt.density_softplus`` change.  None if this tree /
    format renders through kernels that keep no such index."""
    lib = library()
    ct = _pack_tree(tree)
    co = opt._pack()
    lib.svoxb_render_scratch_words.restype = C.c_int64
    words = lib.svoxb_render_scratch_words(C.byref(ct))
    if words <= 0:
        return None
    with torch.cuda.device(tree.data.device):
        scratch = torch.empty(words, dtype=torch.int32, device=tree.data.device)
        st = lib.svoxb_render_scratch_build(C.byref(ct), C.byref(co),
                                            C.c_void_p(scratch.data_ptr()), _stream())
    if st in (3, 4, ERR_TOO_LARGE):      # format / option / size the queue kernels do not take
        return None
    if st:
        _raise(st, "render_scratch_build")
    return scratch


def volume_render(tree, rays, opt, prepared=None):
    """-> (Q, out_dim); svox/csrc/rt_kernel.cu:1019-1036.  ``prepared``: a tensor from
    ``render_scratch`` for the same tree and options (skips the per-call index build)."""
    with _timed("volume_render"):
        return host().volume_render(tree, rays, opt, False, prepared)


def volume_render_image(tree, cam, opt, prepared=None):
    """-> (height, width, out_dim); svox/csrc/rt_kernel.cu:1038-1057.  ``prepared`` as for
    ``volume_render``."""
    return host().volume_render(tree, cam, opt, True, prepared)


# ---------------------------------------------------------------------------
# Logged forward / replay backward (training step without a second march)

_LOG_SLACK_CHUNKS = 2 * 16384   # chunks the forward's warps take and leave partly empty
_items_per_ray = 80.0           # running estimate used to size the item log


class _LogWatch:
    """Learns how large the item log has to be WITHOUT making the host wait for the device.

    After a logged forward the number of chunks it asked for and of samples it wrote (in units
    of 32) are copied to pinned host memory, asynchronously (host.cpp); whenever the next log is
    sized, the counts that have arrived by then adapt the per-ray estimate.  A log that was too
    small costs that one step a marching backward (decided on the device, see
    ``volume_render_backward_replay``), never a wrong gradient."""
    last_used = last_cap = 0

    @classmethod
    def poll(cls, wait=False):
        """Fold the counts that have arrived into the estimate; ``wait`` blocks for all."""
        global _items_per_ray
        if wait and host().logs_pending():
            for dev in range(torch.cuda.device_count()):
                torch.cuda.synchronize(dev)
        for used, batches, n_rays, cap in host().poll_logs():
            cls.last_used, cls.last_cap = used, cap
            if n_rays:
                # items, or the chunks they took beyond the slack: keep 25 % head room
                items = 32 * max(batches, used - _LOG_SLACK_CHUNKS)
                need = max(8.0, 1.25 * items / n_rays)
                _items_per_ray = need if used > cap else max(need, 0.9 * _items_per_ray)
        return _items_per_ray


def log_estimate(wait=False):
    """Current estimate of contributing samples per ray (what the next item log is sized by),
    after folding in the counts of finished forwards; ``wait=True`` waits for all of them."""
    return _LogWatch.poll(wait=wait)


def log_eligible(tree, opt):
    """Whether the logged forward / replay backward pair applies to this call."""
    data = tree.data
    M, N, K = data.shape[0], data.shape[1], data.shape[4]
    layout = K == 4 if opt.format == FORMAT_RGBA else \
        opt.basis_dim in (1, 4, 9, 16, 25) and K == 3 * opt.basis_dim + 1
    return (layout and N == 2 and M < 1 << 28
            and opt.sigma_thresh == 0.0 and opt.stop_thresh == 0.0
            and data.dtype == torch.float32
            # records of whole 16-byte words are read as such
            and (K % 4 != 0 or data.data_ptr() % 16 == 0))


def log_capacity(n_rays):
    """Chunks of the next log for ``n_rays`` rays."""
    return int(n_rays * _LogWatch.poll() / 32) + _LOG_SLACK_CHUNKS


def refuse_tangent(data):
    """Raises for a ``data`` that carries a forward-mode tangent: there is no derivative of that
    kind here, and the calls that make no autograd node would drop it."""
    if _fwd._current_level >= 0 and _fwd.unpack_dual(data).tangent is not None:
        raise NotImplementedError("svox_b200 has no forward-mode derivatives")


def log_words(capacity):
    """int32 words of a log of ``capacity`` chunks."""
    fn = library().svoxb_item_log_words
    fn.restype = C.c_int64
    return fn(C.c_int64(capacity))


def log_is_sorted(tree, n_rays, image):
    """Whether a logged forward of this size sorts its samples, so that the replay clears the
    gradient on the way."""
    return host().log_is_sorted(tree, n_rays, image, log_capacity(n_rays))


def n_rays_of(rays_or_cam, image):
    return rays_or_cam.height * rays_or_cam.width if image else rays_or_cam.origins.shape[0]


def volume_render_logged(tree, rays_or_cam, opt, image=False):
    """Forward render that also records its contributing samples.

    -> (out, (log, capacity_chunks)); pass the pair to ``volume_render_backward_replay``.
    """
    cap = log_capacity(n_rays_of(rays_or_cam, image))
    with _timed("volume_render"):
        out, log = host().volume_render_logged(tree, rays_or_cam, opt, image, cap)
    return out, (log, cap)


def log_chunks_used(log):
    """Chunks the logged forward asked for (synchronises the current stream)."""
    used = C.c_int64(0)
    st = library().svoxb_item_log_used(C.c_void_p(log.data_ptr()), C.byref(used), _stream())
    if st:
        _raise(st, "item_log_used")
    return used.value


def volume_render_backward_replay(tree, rays_or_cam, opt, grad_output, fwd_out, logpair,
                                  image=False, used=0, zeroed=None):
    """Gradient w.r.t. data from the item log of ``volume_render_logged``.

    ``used=0``: the host does not know whether the log was large enough and does not wait to
    find out -- the kernels check on the device, and a marching backward enqueued behind them
    takes over in that case.  ``used`` > 0: a count read with ``log_chunks_used`` that fits
    the capacity (no fallback is enqueued).  ``zeroed``: a zero tensor like
    ``data`` to add the gradient into (else one is made here)."""
    log, cap = logpair
    with _timed("volume_render_backward"):
        return host().volume_render_backward_replay(tree, rays_or_cam, opt, image, grad_output,
                                                    fwd_out, log, cap, used, zeroed)


def volume_render_hessdiag_replay(tree, rays_or_cam, opt, fwd_out, logpair, used, image=False):
    """Gauss-Newton diagonal of the squared error alone, from the item log (third result of the
    reference's ``se_grad``).  ``used``: the count from ``log_chunks_used`` (there is no
    marching fallback for this result, so the caller has to know that the log was large
    enough)."""
    lib = library()
    log, cap = logpair
    dev = tree.data.device
    if not 0 < used <= cap:
        raise RuntimeError("the item log overflowed or its chunk count is not known")
    with torch.cuda.device(dev):
        ct = _pack_tree(tree)
        co = opt._pack()
        _check_input(fwd_out, "fwd_out")
        if fwd_out.numel() != 3 * n_rays_of(rays_or_cam, image):
            raise RuntimeError("fwd_out must have the shape of the render")
        if log.numel() < log_words(cap):
            raise RuntimeError("the item log is smaller than its capacity")
        hess = torch.empty_like(tree.data, memory_format=torch.contiguous_format)
        if image:
            cs = _pack_camera(rays_or_cam, dev)
            fn = lib.svoxb_volume_render_image_hessdiag_replay
        else:
            cs = _pack_rays(rays_or_cam, dev)
            fn = lib.svoxb_volume_render_hessdiag_replay
        st = fn(C.byref(ct), C.byref(cs), C.byref(co), C.c_void_p(fwd_out.data_ptr()),
                C.c_void_p(log.data_ptr()), C.c_int64(cap), C.c_int64(used),
                C.c_void_p(hess.data_ptr()), C.c_int(1), _stream())
    if st:
        _raise(st, "volume_render_hessdiag_replay")
    return hess


# Rays up to which nobody waits to learn whether a log of ``se_grad`` was large enough: its slack
# alone holds 256 samples for each of them.
_SE_GRAD_UNCHECKED = 4096


def se_grad(tree, rays_or_cam, opt, colors, image=False):
    """-> (render, gradient, Gauss-Newton diagonal) of the squared error against ``colors``
    (the reference's ``se_grad``) through the item log.

    A log that was too small: up to ``_SE_GRAD_UNCHECKED`` rays that is noticed on the device,
    where a march enqueued behind the replay takes over.  With more rays that march would take
    some 20 times as long as the call (it adds float by float), so the host looks, while the replay
    runs, and repeats the call with a larger log."""
    n = n_rays_of(rays_or_cam, image)
    cap = log_capacity(n)
    for attempt in range(4):
        if attempt == 1 and tree._weight_accum is not None:     # the weights have been added
            tree = copy.copy(tree)
            tree._weight_accum = None
        out, grad, hess, used = host().se_grad(tree, rays_or_cam, opt, image, colors, cap,
                                               n > _SE_GRAD_UNCHECKED, attempt == 0)
        if used <= cap:
            return out, grad, hess
        if used < 1 << 40:          # (more: given up, not for its size)
            cap = used + used // 4 + _LOG_SLACK_CHUNKS
    grad, hess = se_grad_march(tree, rays_or_cam, opt, out,
                               colors.reshape(out.shape).contiguous(), image=image)
    return out, grad, hess


def se_grad_march(tree, rays_or_cam, opt, fwd_out, colors, image=False):
    """-> (grad, hessdiag) of the squared error ``1/2 sum (fwd_out - colors)^2`` by marching
    the rays once more: any record layout with at most four output channels.  ``fwd_out``: the
    render of the same inputs with both thresholds zero."""
    lib = library()
    dev = tree.data.device
    with torch.cuda.device(dev):
        ct = _pack_tree(tree)
        co = opt._pack()
        _check_input(fwd_out, "fwd_out")
        _check_input(colors, "colors")
        if colors.numel() != fwd_out.numel():
            raise RuntimeError("colors must have the shape of the render")
        grad = torch.zeros_like(tree.data, memory_format=torch.contiguous_format)
        hess = torch.zeros_like(grad)
        if image:
            cs = _pack_camera(rays_or_cam, dev)
            fn = lib.svoxb_se_grad_image_march
        else:
            cs = _pack_rays(rays_or_cam, dev)
            fn = lib.svoxb_se_grad_march
        st = fn(C.byref(ct), C.byref(cs), C.byref(co), C.c_void_p(fwd_out.data_ptr()),
                C.c_void_p(colors.data_ptr()), C.c_void_p(grad.data_ptr()),
                C.c_void_p(hess.data_ptr()), C.c_int(0), _stream())
    if st:
        _raise(st, "se_grad_march")
    return grad, hess


def allreduce_multimem(multicast_ptr, n_floats, rank, world):
    """Sum ``n_floats`` floats over the GPUs of a multicast object, in place, on the current
    stream (see ``svoxb_allreduce_multimem``); the caller provides the barriers around it."""
    st = library().svoxb_allreduce_multimem(C.c_void_p(int(multicast_ptr)), C.c_int64(n_floats),
                                            C.c_int(rank), C.c_int(world), _stream())
    if st:
        _raise(st, "allreduce_multimem")


def replay_part_ranges(M, K, n_parts):
    """Leaf-slot ranges [(begin, end)] of the ``n_parts`` parts of a replay backward for a tree
    of ``M`` nodes with ``K`` floats per record (whole bins; the same on every process)."""
    shift = library().svoxb_replay_bin_shift(C.c_int64(M), C.c_int32(K))
    n_slots = M * 8
    n_bins = ((n_slots - 1) >> shift) + 1
    cut = [min(((p * n_bins) // n_parts) << shift, n_slots) for p in range(n_parts)] + [n_slots]
    return list(zip(cut[:-1], cut[1:]))


def volume_render_backward_replay_parts(tree, rays_or_cam, opt, grad_output, fwd_out, logpair,
                                        n_parts, on_part, reserve_sms=0, image=False,
                                        zeroed=None):
    """The replay backward in ``n_parts`` consecutive leaf ranges.  After each part
    ``on_part(rows)`` is called with the flat view of the gradient rows that are final
    (e.g. to start their all-reduce while the next part is computed).  The host never waits
    for the device: whether the log was large enough is decided there, and the marching
    fallback runs before the first part, so the rows handed on are final either way and every
    process of a data-parallel job makes the same ``on_part`` calls."""
    lib = library()
    log, cap = logpair
    dev = tree.data.device
    K = tree.data.shape[-1]
    with torch.cuda.device(dev):
        ct = _pack_tree(tree)
        co = opt._pack()
        _check_input(grad_output, "grad_output")
        _check_input(fwd_out, "fwd_out")
        n = n_rays_of(rays_or_cam, image)
        if grad_output.numel() != 3 * n or fwd_out.numel() != 3 * n:
            raise RuntimeError("grad_output and fwd_out must have the shape of the render")
        if log.numel() < log_words(cap):
            raise RuntimeError("the item log is smaller than its capacity")
        if image:
            cs = _pack_camera(rays_or_cam, dev)
            begin = lib.svoxb_replay_image_begin
        else:
            cs = _pack_rays(rays_or_cam, dev)
            begin = lib.svoxb_replay_begin
        grad = zeroed if zeroed is not None else \
            torch.zeros_like(tree.data, memory_format=torch.contiguous_format)
        flat = grad.view(-1)
        ranges = replay_part_ranges(ct.M, K, n_parts)
        job = C.c_void_p(None)
        with _timed("volume_render_backward"):
            st = begin(C.byref(ct), C.byref(cs), C.byref(co),
                       C.c_void_p(grad_output.data_ptr()), C.c_void_p(fwd_out.data_ptr()),
                       C.c_void_p(log.data_ptr()), C.c_int64(cap), C.c_int64(0),
                       C.c_int(n_parts), C.c_void_p(grad.data_ptr()), _stream(), C.byref(job))
            if st:
                _raise(st, "replay_begin")
            try:
                lo, hi = C.c_int64(0), C.c_int64(0)
                for part in range(n_parts):
                    st = lib.svoxb_replay_scatter(job, C.c_int(part), C.c_void_p(grad.data_ptr()),
                                                  C.c_int(reserve_sms), _stream())
                    if st:
                        _raise(st, "replay_scatter")
                    lib.svoxb_replay_part_range(job, C.c_int(part), C.byref(lo), C.byref(hi))
                    assert (lo.value, hi.value) == ranges[part]
                    on_part(flat[lo.value * K:hi.value * K])
            finally:
                lib.svoxb_replay_end(job, _stream())
    return grad


def volume_render_backward(tree, rays, opt, grad_output, fwd_out=None):
    """-> gradient w.r.t. data (like data); svox/csrc/rt_kernel.cu:1059-1083.

    ``fwd_out`` (optional, not in the reference signature) is the forward
    result for the same inputs; it lets the kernel march each ray once.
    """
    with _timed("volume_render_backward"):
        return host().volume_render_backward(tree, rays, opt, False, grad_output, fwd_out)


def volume_render_image_backward(tree, cam, opt, grad_output, fwd_out=None):
    """-> gradient w.r.t. data; svox/csrc/rt_kernel.cu:1085-1109."""
    return host().volume_render_backward(tree, cam, opt, True, grad_output, fwd_out)


def march_stats(tree, rays, opt):
    """Per-ray (visits, contributing samples forward, contributing samples backward),
    three (Q,) int32 tensors (no counterpart in the reference)."""
    lib = library()
    ct = _pack_tree(tree)
    cr = _pack_rays(rays, tree.data.device)
    co = opt._pack()
    with torch.cuda.device(tree.data.device):
        outs = [torch.zeros(cr.Q, dtype=torch.int32, device=tree.data.device) for _ in range(3)]
        st = lib.svoxb_march_stats(C.byref(ct), C.byref(cr), C.byref(co),
                                   *[C.c_void_p(t.data_ptr()) for t in outs], _stream())
    if st:
        _raise(st, "march_stats")
    return tuple(outs)


def device_status(clear=True):
    """Synchronise and return the device anomaly word (0 = none), see svox_b200.h."""
    return int(library().svoxb_device_status(C.c_int(int(clear)), _stream()))


def check_device_status():
    st = device_status(clear=True)
    if st:
        _raise(st, "device_status")


def reserve_sms(n):
    """Leave ``n`` multiprocessors to other kernels (a collective on another stream) in the
    library's persistent kernels; returns the previous setting (``n < 0``: query only)."""
    return int(library().svoxb_reserve_sms(C.c_int(int(n))))


def version():
    return library().svoxb_version().decode()
