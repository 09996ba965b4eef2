"""Fused multi-view rendering of a Universal Beta Splatting scene (GB300 path).

One call renders a batch of views, of any mix of resolutions and timestamps,
with five stream-ordered launches (per-primitive forward, scan, emit, bucket
sort, blend) and one autograd node whose backward is two launches (blend
backward, per-primitive backward).  The mathematics is the reference model's
render (scene/beta_model.py:660-722 + rendering.py:17-232), evaluated per
(view, primitive): each primitive is conditioned on the ray to that view's
camera (and its timestamp), so views are consistent with rendering them one at
a time.

    from ubs.render import Renderer, Views
    r = Renderer(dim=6)
    views = Views([cam0, cam1], device="cuda")      # ubs.scene.Camera objects
    colors, alphas = r.render(params, views)       # flat [P, 3], [P]
    images = views.split(colors)                   # list of [H, W, 3]
"""
import contextlib
import ctypes
import threading
import weakref
from typing import Dict, List, Optional, Sequence

import torch

from . import _lib as L

PARAM_ORDER = ("xyz", "mean", "scale", "l_triangle", "opacity", "beta", "rgb")
STATUS_OVERFLOW = 4
STATUS_NEG_DEPTH = 2
MAX_CAPACITY = 2 ** 31 - 1  # intersections of one call (their positions are int32)


class Views:
    """Cameras of one render call, flattened into (view, tile) buckets and one
    pixel buffer.  `cameras` are ubs.scene.Camera objects (viewmat, K, width,
    height, timestamp).  The per-view tables go to the device in one copy from
    a pinned staging buffer, on `stream` (default: the current one)."""

    def __init__(self, cameras: Sequence, tile_size: int = 16, device=None, stream=None):
        if len(cameras) == 0:
            raise ValueError("need at least one view")
        device = torch.device(device or cameras[0].viewmat.device)
        C = len(cameras)
        # the camera centre the reference model conditions on: the camera's
        # own value (computed where its matrices live), so the view-direction
        # queries round the same way
        centers = []
        for c in cameras:
            center = getattr(c, "position", None)
            centers.append(getattr(c, "center", None) if center is None else center)
        (staging, self.viewmats, self.intr, self.centers, self.times, self.dims, self.tile_base,
         self.pix_base, tile_base, pix_base) = L.untraced(
             "pack_views", [c.viewmat for c in cameras], [c.K for c in cameras], centers,
             [float(c.timestamp) for c in cameras], [c.width for c in cameras],
             [c.height for c in cameras], tile_size, device,
             None if stream is None else (stream.stream_id, stream.device_index))
        self.C = C
        self.tile_size = tile_size
        self.shapes = [(c.height, c.width) for c in cameras]
        self.n_buckets = tile_base[-1]
        self.n_pixels = pix_base[-1]
        self.pix_base_host = pix_base
        self.device = device
        self._staging = staging  # the pinned buffer must outlive the copy

    def _tables(self):
        return [self.viewmats, self.intr, self.centers, self.times, self.dims, self.tile_base,
                self.pix_base]

    def split(self, flat: torch.Tensor) -> List[torch.Tensor]:
        """Per-view [H, W, ...] views of a flat per-pixel buffer."""
        out = []
        for v, (h, w) in enumerate(self.shapes):
            a, b = self.pix_base_host[v], self.pix_base_host[v + 1]
            out.append(flat[a:b].view(h, w, *flat.shape[1:]))
        return out

    def join(self, images: Sequence[torch.Tensor]) -> torch.Tensor:
        """Inverse of split: per-view [H, W, ...] tensors -> flat [P, ...]."""
        return torch.cat([im.reshape(-1, *im.shape[2:]) for im in images], 0)


class Renderer:
    """Renders scenes through the fused path and keeps the intersection
    capacity of its workspaces.  `exact_cond_grad` selects the exact
    conditioning gradient instead of the reference's backward formula."""

    def __init__(self, dim: int = 6, tile_size: int = 16, eps2d: float = 0.3,
                 near_plane: float = 0.01, far_plane: float = 1e10, radius_clip: float = 0.0,
                 capacity: Optional[int] = None, exact_cond_grad: bool = False):
        if dim not in (6, 7):
            raise ValueError("dim must be 6 or 7")
        self.dim = dim
        self.tile_size = tile_size
        self.eps2d, self.near, self.far, self.radius_clip = eps2d, near_plane, far_plane, radius_clip
        self.capacity = capacity
        self.exact_cond_grad = exact_cond_grad
        self.last_isects = None
        self._pending = None  # (stats, capacity) of an unchecked frame
        self.last_ws, self.last_cap = None, None

    # ---------------------------------------------------------------- helpers
    def _check_pending(self):
        if self._pending is None:
            return
        stats, cap = self._pending
        self._pending = None
        T, status = stats.wait()
        self.last_isects = T
        if status & STATUS_NEG_DEPTH:
            raise RuntimeError("scene render: a visible primitive has a negative depth")
        if status & STATUS_OVERFLOW or T > cap:
            self.capacity = max(self.capacity or 0, int(T * 1.25) + 1024)
            raise RuntimeError("scene render: an earlier unchecked frame needed %d intersections "
                               "but had capacity %d; capacity is now %d" % (T, cap, self.capacity))
        if T > cap - cap // 8:
            # a scene that grows from frame to frame (training) gets its room
            # before a frame overflows, as far as a capacity goes
            self.capacity = max(self.capacity or 0, min(int(T * 1.25) + 1024, MAX_CAPACITY))

    def stats(self):
        """(intersections, status bits) of the last forward's workspace; raises
        if that frame overflowed its capacity.  Synchronises the stream."""
        import ctypes
        T, status = ctypes.c_int64(0), ctypes.c_uint32(0)
        L.call("ubs_scene_stats", L.ptr(self.last_ws), ctypes.byref(T), ctypes.byref(status),
               L.stream(self.last_ws.device))
        self.last_isects = int(T.value)
        if status.value & STATUS_NEG_DEPTH:
            raise RuntimeError("scene render: a visible primitive has a negative depth")
        if status.value & STATUS_OVERFLOW or T.value > self.last_cap:
            self.capacity = max(self.capacity or 0, int(T.value * 1.25) + 1024)
            raise RuntimeError("scene render: a frame needed %d intersections but had capacity "
                               "%d; capacity is now %d" % (T.value, self.last_cap, self.capacity))
        return int(T.value), int(status.value)

    def workspace_bytes(self, C, N, n_buckets, capacity):
        return L.query("ubs_scene_workspace_bytes", C, N, n_buckets, capacity)

    def radii(self, views: Views, N: int):
        """The last forward's per-(view, primitive) radii, int32 [C, N] (a view
        into its workspace; 0 where a primitive was not rendered)."""
        import ctypes
        r, d = ctypes.c_int64(), ctypes.c_int64()
        L.call("ubs_scene_workspace_offsets", views.C, N, views.n_buckets, self.last_cap,
               ctypes.byref(r), ctypes.byref(d))
        n = views.C * N
        return self.last_ws[r.value:r.value + 4 * n].view(torch.int32).view(views.C, N)

    def _sections(self, views: Views, N: int):
        """Byte offsets of the last forward's workspace sections
        (ubs_scene_workspace_layout: records, radii, depths, bucket starts,
        keys)."""
        secs = (ctypes.c_int64 * 5)()
        L.call("ubs_scene_workspace_layout", views.C, N, views.n_buckets, self.last_cap, secs, 5)
        return [int(x) for x in secs]

    def projected(self, views: Views, N: int):
        """The last forward's per-(view, primitive) projection, as the
        reference's meta entries: dict of means2d [C, N, 2], conics [C, N, 3],
        opacities [C, N] (conditioned), betas [C, N], radii int32 [C, N],
        depths [C, N] (views into the workspace; zeros where the radius is 0)."""
        rec, rad, dep, _, _ = self._sections(views, N)
        n = views.C * N
        r = self.last_ws[rec:rec + 32 * n].view(torch.float32).view(views.C, N, 8)
        return {"means2d": r[..., 0:2], "opacities": r[..., 2], "betas": r[..., 3],
                "conics": r[..., 4:7],
                "radii": self.last_ws[rad:rad + 4 * n].view(torch.int32).view(views.C, N),
                "depths": self.last_ws[dep:dep + 4 * n].view(torch.float32).view(views.C, N)}

    def intersections(self, views: Views, N: int):
        """The last forward's sorted intersections in the reference's layout,
        one entry per view: (isect_ids int64 [T_v] = tile << 32 | depth bits,
        flatten_ids int32 [T_v] = primitive index, isect_offsets int32
        [th, tw]) -- what isect_tiles + isect_offset_encode return for that
        view alone (isect_tiles.cu:82-96, 287-367).  Reads the intersection
        count (synchronises)."""
        T, _ = self.stats()
        _, _, _, o_off, o_key = self._sections(views, N)
        nb = views.n_buckets
        # bucket starts (exclusive scan of the counts); the end of the last
        # bucket is the intersection total
        starts = self.last_ws[o_off:o_off + 4 * nb].view(torch.int32).long()
        ends = torch.cat([starts[1:], starts.new_full((1,), T)])
        keys = self.last_ws[o_key:o_key + 8 * T].view(torch.int64)
        tb = views.tile_base.long().cpu()
        out = []
        for v in range(views.C):
            b0, b1 = int(tb[v]), int(tb[v + 1])
            a, b = int(starts[b0]), int(ends[b1 - 1])
            k = keys[a:b]
            counts = ends[b0:b1] - starts[b0:b1]
            tile = torch.repeat_interleave(torch.arange(b1 - b0, device=k.device), counts)
            ids = (tile << 32) | ((k >> 32) & 0xffffffff)
            fl = ((k & 0xffffffff) - v * N).to(torch.int32)
            h, w = views.shapes[v]
            ts = views.tile_size
            th, tw = (h + ts - 1) // ts, (w + ts - 1) // ts
            out.append((ids, fl, (starts[b0:b1] - a).to(torch.int32).view(th, tw)))
        return out

    def forward_raw(self, p: Dict[str, torch.Tensor], views: Views, bg, check=True,
                    prim_mask=None, color_mode=0, image=None):
        """Run the forward kernels; returns (colors, alphas, last_ids, workspace, capacity).

        check=True reads the intersection count back (synchronising) and
        re-runs an overflowing frame; check=False reads it back
        asynchronously and reports an overflow at the next call; check="none"
        issues nothing but the kernels (safe inside CUDA graph capture) and
        leaves the verification to `stats()` after the frame(s).
        prim_mask (uint8 [N]) leaves out primitives whose entry is 0;
        color_mode=1 renders depth into channel 0 (one view, no backward).
        image (pinned float32 host tensor of 3 * n_pixels values) takes the
        colours and is returned as such; it is complete once the current stream
        has been waited for."""
        return self._forward([p[k] for k in PARAM_ORDER], views, bg, check, prim_mask, color_mode,
                             False, image)

    def _forward(self, tensors, views, bg, check, prim_mask, color_mode, grad, image=None):
        if check == "none":
            if self.capacity is None:
                raise RuntimeError("check='none' needs a capacity (render once with check=True)")
        else:
            self._check_pending()
        N = tensors[0].shape[0]
        # first frame: a guess from the pixel count (re-run below if too small)
        cap = self.capacity or max(1 << 16, min(16 * N * views.C, 8 * views.n_pixels))
        native = L.native()
        while True:
            call = native.SceneCall(self.dim, views._tables(), views.n_buckets, views.n_pixels,
                                    self.tile_size, self.eps2d, self.near, self.far,
                                    self.radius_clip, bool(self.exact_cond_grad), cap)
            colors, alphas, last, ws, stats = native.scene_forward(
                call, tensors, bg, prim_mask, color_mode, check != "none", grad, image)
            self.last_ws, self.last_cap = ws, cap
            if check == "none":
                return colors, alphas, last, ws, cap
            if not check:
                self._pending = (stats, cap)
                return colors, alphas, last, ws, cap
            T, status = stats.wait()
            self.last_isects = T
            if status & STATUS_NEG_DEPTH:
                raise RuntimeError("scene render: a visible primitive has a negative depth")
            if T <= cap:
                if self.capacity is None:
                    self.capacity = max(int(T * 1.25) + 1024, 1 << 16)
                return colors, alphas, last, ws, cap
            cap = int(T * 1.25) + 1024
            self.capacity = cap

    def render(self, params: Dict[str, torch.Tensor], views: Views,
               backgrounds: Optional[torch.Tensor] = None, check=True):
        """Differentiable render of all views: colors [P, 3], alphas [P].
        `check`: True, False or "none", as for forward_raw."""
        if backgrounds is None:
            bg = torch.zeros(views.C, 3, device=params["xyz"].device)
        else:
            bg = backgrounds.reshape(-1, 3).expand(views.C, 3).contiguous().float()
        tensors = [params[k] for k in PARAM_ORDER]
        if L.tracing():
            return L.recorded("scene_render", lambda bg, *p: self._forward(
                p, views, bg, check, None, 0, True)[:2], bg, *tensors)
        colors, alphas, _, _, _ = self._forward(tensors, views, bg, check, None, 0, True)
        return colors, alphas


class _Graphs:
    """Destroying a graph is not permitted while another is being captured and
    fails that capture; a step in a reference cycle can die at any time, inside
    a later step's capture too (a cycle collection there).  The graphs of steps
    that die during a capture, on whatever thread, are kept until the last
    capture has ended."""

    def __init__(self):
        self._lock = threading.RLock()  # a collection may run while it is held
        self._captures, self._kept = 0, []

    def release(self, graph):
        with self._lock:
            if self._captures:
                self._kept.append(graph)

    @contextlib.contextmanager
    def capturing(self):
        with self._lock:
            self._captures += 1
        try:
            yield
        finally:
            kept = []
            with self._lock:
                self._captures -= 1
                if not self._captures:
                    kept, self._kept = self._kept, kept
            del kept  # destroyed here


_GRAPHS = _Graphs()


class GraphedStep:
    """One training step -- fused render of `views`, `loss_fn(colors, alphas)`,
    backward to every parameter -- captured once into a CUDA graph and then
    replayed with a single launch.

    The parameters must keep their storage between replays (update them in
    place, e.g. with an optimizer or `copy_`); after each replay their `.grad`
    tensors (owned by the graph's memory pool) hold that step's gradients and
    `loss` holds its value.  The intersection capacity is fixed when the step
    is captured (the first frame's count times `headroom`); `check()` reads the
    last replay's count back and raises if the frame overflowed, in which case
    the step must be captured again.  Capture on parameter tensors that have
    not been through an eager backward on the default stream (or on fresh
    copies of them): PyTorch's gradient accumulation for such leaves would
    make the capture wait on that stream, which capture does not allow.

    With `optimizer` (ubs.optim.FusedAdam) the optimizer's update is captured
    too: the gradients then keep fixed storage (allocated while warming up,
    zeroed inside the graph) and `replay()` runs the optimizer's host part
    (`prepare()`) before launching the graph."""

    def __init__(self, renderer: Renderer, params: Dict[str, torch.Tensor], views: Views,
                 backgrounds: Optional[torch.Tensor], loss_fn, headroom: float = 1.5,
                 warmup: int = 3, before_capture=None, optimizer=None):
        self.r, self.p, self.views, self.loss_fn = renderer, params, views, loss_fn
        dev = params["xyz"].device
        self.bg = (torch.zeros(views.C, 3, device=dev) if backgrounds is None
                   else backgrounds.reshape(-1, 3).expand(views.C, 3).contiguous().float())
        with torch.no_grad():
            renderer.render(params, views, self.bg, check=True)
        renderer.capacity = int(renderer.last_isects * headroom) + 4096
        self.optimizer = optimizer
        side = torch.cuda.Stream(dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            for _ in range(warmup):
                for v in params.values():
                    v.grad = None
                self._body()
                if optimizer is not None:
                    optimizer.step()
        torch.cuda.current_stream(dev).wait_stream(side)
        if optimizer is None:
            for v in params.values():
                v.grad = None
        if before_capture is not None:
            before_capture()
        self.graph = torch.cuda.CUDAGraph()
        n0 = L.query("ubs_launch_count")
        # the graph outlives this object until no step is being captured
        weakref.finalize(self, _GRAPHS.release, self.graph).atexit = False
        with _GRAPHS.capturing(), torch.cuda.graph(self.graph):
            if optimizer is not None:
                for v in params.values():
                    v.grad.zero_()
            self.loss = self._body()
            if optimizer is not None:
                optimizer.launch()
        # library kernels in the graph (each replay launches them all)
        self.launches_per_replay = int(L.query("ubs_launch_count") - n0)

    def _body(self):
        colors, alphas = self.r.render(self.p, self.views, self.bg, check="none")
        loss = self.loss_fn(colors, alphas)
        loss.backward()
        return loss

    def replay(self):
        if self.optimizer is not None:
            self.optimizer.prepare()
        self.graph.replay()
        return self.loss

    def check(self):
        return self.r.stats()


class HostFedStep:
    """Steps whose inputs come from pinned host memory every step (a data
    loader, another process, a parameter store), with the copies of step k+1
    overlapping the compute of step k.

    `make_inputs()` returns (params, feeds, loss_fn): the parameter tensors
    of a GraphedStep, the device tensors that receive the host data each step
    (any of the parameters and, e.g., a target image the loss reads), and
    the loss over (colors, alphas).  It is called `depth` times (default 2):
    each buffer set gets its own tensors and its own captured step.
    `step(host)` copies host[i] (pinned, same shapes as feeds[i]) into the
    next set's feeds on a copy stream once that set's previous step is done,
    replays the set's graph on the current stream once the copies are done,
    and copies the loss into a pinned slot; `losses()` waits for the device
    and returns the values of the steps since the last call.  `start()` makes
    the copy stream wait for the current stream's work issued so far (call it
    where a timed region begins)."""

    def __init__(self, renderer: Renderer, views: Views, backgrounds, make_inputs,
                 depth: int = 2, headroom: float = 1.5, warmup: int = 3):
        if depth < 1:
            raise ValueError("depth must be >= 1")
        self.sets = []
        for _ in range(depth):
            params, feeds, loss_fn = make_inputs()
            gs = GraphedStep(renderer, params, views, backgrounds, loss_fn, headroom, warmup)
            self.sets.append((gs, list(feeds)))
        self.device = self.sets[0][1][0].device
        self.copy_stream = torch.cuda.Stream(self.device)
        self.copied = [torch.cuda.Event() for _ in range(depth)]
        self.done = [None] * depth
        self.ring = 256
        self.loss_host = torch.empty(self.ring, pin_memory=True)
        self.k = 0
        self.pending = []
        self.launches_per_step = self.sets[0][0].launches_per_replay

    def start(self):
        ev = torch.cuda.Event()
        ev.record(torch.cuda.current_stream(self.device))
        self.copy_stream.wait_event(ev)

    def step(self, host: Sequence[torch.Tensor]):
        s = self.k % len(self.sets)
        gs, feeds = self.sets[s]
        if len(host) != len(feeds):
            raise ValueError("step() needs one host tensor per feed")
        cs = self.copy_stream
        cur = torch.cuda.current_stream(self.device)
        if self.done[s] is not None:
            cs.wait_event(self.done[s])  # the set's previous step has read its inputs
        with torch.cuda.stream(cs), torch.no_grad():
            for dst, src in zip(feeds, host):
                dst.copy_(src, non_blocking=True)
        self.copied[s].record(cs)
        cur.wait_event(self.copied[s])
        loss = gs.replay()
        slot = self.k % self.ring
        if len(self.pending) == self.ring:
            raise RuntimeError("call losses() at least every %d steps" % self.ring)
        self.loss_host[slot:slot + 1].copy_(loss.detach().view(1), non_blocking=True)
        ev = torch.cuda.Event()
        ev.record(cur)
        self.done[s] = ev
        self.pending.append(slot)
        self.k += 1
        return slot

    def losses(self) -> List[float]:
        torch.cuda.current_stream(self.device).synchronize()
        out = [float(self.loss_host[i]) for i in self.pending]
        self.pending = []
        return out

    def check(self):
        return [gs.check() for gs, _ in self.sets]
