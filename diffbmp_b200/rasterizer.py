"""Torch-facing host layer over libdbmp.so.

PyTorch supplies device memory and streams; every computation is one of the
library's CUDA kernels.  Tensors must be CUDA tensors; nothing here falls
back to a CPU or PyTorch implementation.

Main objects:

* ``Atlas``       -- a template atlas resident on the device in one storage
                     kind (f32 reference layout, or f32/f16/bf16 bilinear quads)
                     plus its per-template content bboxes.
* ``Rasterizer``  -- one canvas (H, W, tile size): binning, forward, backward
                     and the fused fit step; owns the scratch it reuses.
* ``rasterize``   -- autograd entry point (``RasterizeFunction``).
"""
from __future__ import annotations

import contextlib
import ctypes
from dataclasses import dataclass
from typing import Optional

import torch

from . import _lib
from ._lib import (ATLAS_BF16_PAIR, ATLAS_BF16_QUAD, ATLAS_F16_PAIR, ATLAS_F16_QUAD, ATLAS_F32, ATLAS_F32_QUAD,
                   BIN_CONTENT, BIN_CONTENT_REF, BIN_CULL, EXTENDED_ATLAS, FOLLOWED_ATLAS, Canvas, DbmpError,
                   FollowedCanvas, call, lib)

# Atlas storage kinds: "f32" is the reference layout; the precision form
# stores half / bfloat16 texels as horizontal pairs ("f16", "bf16", two 4-byte
# loads per bilinear sample) or as full bilinear quads ("f16q", "bf16q", "f32q").
KIND_NAMES = {"f32": ATLAS_F32, "f32q": ATLAS_F32_QUAD, "f16q": ATLAS_F16_QUAD, "bf16q": ATLAS_BF16_QUAD,
              "f16": ATLAS_F16_PAIR, "bf16": ATLAS_BF16_PAIR}

# The renders of an "f32" atlas walk a copy of its templates packed as f32 quads (16
# bytes a texel) up to this many bytes.  The walks are as fast on quads far beyond
# the L2 as inside it (2048x2048, N=20000, 1024 templates of 256x256, 1 GiB of quads: forward 257 us,
# backward 384, against 549 and 810 on the reference layout; with 16 templates 239
# and 363 against 537 and 800), so the limit only bounds their memory and the time
# to pack them (1.6 ms per GiB).
MAX_F32_QUAD_BYTES = 1 << 30

DEFAULT_T_STOP = 1e-6   # image error <= t_stop * max colour, well inside the 1e-5 parity bar


def _ptr(t: Optional[torch.Tensor]):
    return t.data_ptr() if t is not None else None


def _stream(stream=None):
    if stream is not None:
        return stream.cuda_stream
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


_HERE = contextlib.nullcontext()


def _on(stream):
    """The stream as the current one (None: as it is, at none of the cost)."""
    return _HERE if stream is None else torch.cuda.stream(stream)


def _need_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise ValueError("diffbmp_b200 kernels need CUDA tensors (no CPU fallback exists)")


def _f32(t: torch.Tensor) -> torch.Tensor:
    return t.detach().to(torch.float32).contiguous()


def _operand(t: torch.Tensor) -> torch.Tensor:
    """t as a kernel operand: itself where it is contiguous f32 already."""
    return t if t.dtype is torch.float32 and t.is_contiguous() else _f32(t)


def quads_pay(pixels: int, N: int, texels: int) -> bool:
    """Whether the walks of one forward and backward, or of one fit step, of N
    primitives on `pixels` pixels gain more on a packed copy of an "f32" atlas than
    packing it takes, as a job whose templates change on every call pays for it.

    Packing takes 10 us for 64x64 texels, 23 for 8 of 128x128, 61 for 16 of 256x256 and
    10 more for each further million; the walks gain with the pixels and, between 50
    and about 500 primitives, where a pixel is opaque, with their depth.  Forward and
    backward's gain in us on both sides of the line, measured with launches of their
    own for the comparison (5 us more than it takes now):
      one 64x64 (10):     N=200  500x512 0, 768x768 4;  N=300  384x384 -2, 500x512 6
      4 of 64x64 (10):    N=200  384x384 0;  N=300  500x512 11
      8 of 128x128 (23):  N=300  384x384 4, 500x512 15, 600x600 22, 768x768 36;
                          N=600  300x300 18, 384x384 20, 500x512 41
      16 of 256x256 (61): N=60   1500x1500 7;  N=300  500x512 29, 768x768 56,
                          1024x1024 93;  N=600  384x384 29, 600x600 77
      16 of 512x512 (101), 1024x1024 (228): N=600  512x512 52 and 30, 1024x1024 211
                          and 208, 2048x2048 679 and 855"""
    million = 1 << 20
    line = 125_000 + min(texels, million) // 8 + max(0, texels - million) // 9
    return pixels * (min(N, 500) - 50) >= 450 * line


def fit_quads_pay(pixels: int, N: int, texels: int) -> bool:
    """Whether a fit, whose steps share one packed copy, walks quads of an "f32" atlas.

    From 200 primitives on a step gains more than its comparison takes: -5 to 1 us
    with N=60 (8 at 1500x1500), -3 to 15 up to 1024x1024 with 100, 0.7 to 51 with 200,
    4 to 155 with 600, over canvases from 64x64 and atlases from 64x64 to 16 of
    256x256.  The comparison of larger atlases takes that back on small canvases: with
    four million texels, N=600, a step gains -34 us at 64x64, 3 at 256x256 and 23 at
    384x384; with 17 million 5 at 384x384 and 47 at 512x512 (N=200: -17 and -3); with
    67 million 52 at 512x512 and 191 at 1024x1024 (-36 and 7)."""
    return N >= 200 and texels <= (1 << 20) + 64 * pixels


class Filled:
    """Device memory that one stream fills once and calls on any stream then read.
    Made where the fill has just been enqueued on the current stream."""

    def __init__(self, tensor: torch.Tensor):
        self.tensor = tensor
        s = torch.cuda.current_stream(tensor.device)
        self._device, self._home = s.device_index, s.cuda_stream
        self._event = torch.cuda.Event()
        self._event.record(s)
        self._done = False

    def use(self, stream=None) -> torch.Tensor:
        """The tensor, for work enqueued on `stream` (default: the current one) after
        this call: behind the fill, and not freed before that work is done.  Under
        graph capture the caller has waited for the fill, as for the capture's
        other inputs."""
        h = stream.cuda_stream if stream is not None else torch._C._cuda_getCurrentRawStream(self._device)
        if h != self._home:
            s = stream if stream is not None else torch.cuda.current_stream(self.tensor.device)
            if not torch.cuda.is_current_stream_capturing():
                if not self._done:
                    self._done = self._event.query()
                if not self._done:
                    s.wait_event(self._event)
            self.tensor.record_stream(s)
        return self.tensor

    def __reduce__(self):       # (copied and pickled with its owner)
        return Filled, (self.use(),)


class Atlas:
    """Template atlas on the device.  ``templates``: (P,Ht,Wt) or (Ht,Wt).
    ``sigma`` > 0 renders with Gaussian-blurred templates while the content
    bboxes (binning) stay those of the unblurred ones, as the reference's
    VectorRenderer does (vector_renderer.py:80-104).

    An "f32" atlas renders the memory of ``data``, which is the caller's tensor where
    that is contiguous f32, as it is when a call's turn on its stream comes,
    whoever has written to it (quads() packs a copy for the walks, and every
    walk compares it with ``data`` first).  The other kinds hold a packed copy
    made here."""

    def __init__(self, templates: torch.Tensor, kind: str | int = "f32", sigma: float = 0.0):
        t = templates if templates.dim() == 3 else templates.unsqueeze(0)
        _need_cuda(t)
        self.templates = _f32(t)
        self.sigma = float(sigma)
        self.P, self.Ht, self.Wt = (int(v) for v in self.templates.shape)
        self.kind = KIND_NAMES[kind] if isinstance(kind, str) else int(kind)
        st = _stream()
        self.bbox = torch.empty((self.P, 4), dtype=torch.float32, device=t.device)
        call("dbmp_template_bboxes", _ptr(self.templates), self.P, self.Ht, self.Wt, _ptr(self.bbox), st)
        if self.sigma > 0.0:
            blurred = torch.empty_like(self.templates)
            call("dbmp_template_blur", _ptr(self.templates), self.P, self.Ht, self.Wt, ctypes.c_float(self.sigma),
                 _ptr(blurred), st)
            self.templates = blurred
        # an extended atlas (dbmp_atlas_pack_extended) holds the grids, and for
        # "f32" the quads, that let the walks skip work
        self.extended = self.kind != ATLAS_F32 or (self.templates.numel() * 16 <= MAX_F32_QUAD_BYTES
                                                   and not self.templates.is_inference())
        self.own = self.kind != ATLAS_F32     # data is an extended atlas's buffer
        self._quads = None                    # ("f32") Filled extended atlas, version of data that it was packed from
        self._anew = self._anew_next = 0      # calls that pack whatever the version; how many after the next miss
        self.fills = 0                        # (own) how often pack() has filled the buffer
        if self.own:
            self._alloc()
            self.pack(self.templates, st)
        else:
            self.data = self.templates

    def _alloc(self):
        """The extended atlas's buffer; data is the part dbmp_atlas_bytes counts."""
        total = int(lib.dbmp_atlas_extended_bytes(self.P, self.Ht, self.Wt, self.kind))
        buf = torch.empty(total, dtype=torch.uint8, device=self.templates.device)
        self.data = buf[:int(lib.dbmp_atlas_bytes(self.P, self.Ht, self.Wt, self.kind))]
        if self.kind == ATLAS_F32:
            self.data = self.data.view(torch.float32).view(self.P, self.Ht, self.Wt)

    def refresh(self):
        """Has an "f32" atlas packed anew by its next render.  Never needed for the
        result: a render that finds ``data`` changed repeats itself on it, and the
        other walks read it in the reference layout, which is slower.  A change that
        PyTorch counts (``data._version``) is packed anew without this call; writes
        through ``.data``, of another library's kernel or a replayed graph are not
        counted."""
        self._quads = None

    def _missed(self):
        """A render has found the copy out of date and repeats itself: the next ones
        pack anew, one after the first such miss, up to 63 when misses go on."""
        self._quads = None
        self._anew, self._anew_next = self._anew_next, min(2 * self._anew_next + 1, 63)

    def quads(self, stream=None) -> Optional[Filled]:
        """An "f32" atlas's extended copy (quads and grids) for work on `stream`, or
        None where it has none and walks data itself.  A copy never changes once
        packed: calls in flight on other streams or threads keep the one that they
        took."""
        if self.own or not self.extended:
            return None
        q, version = self._quads or (None, -1)
        if self._anew or version != self.data._version:
            self._anew = max(0, self._anew - 1)
            version = self.data._version
            with _on(stream):
                buf = torch.empty(int(lib.dbmp_atlas_extended_bytes(self.P, self.Ht, self.Wt, self.kind)),
                                  dtype=torch.uint8, device=self.data.device)
                call("dbmp_atlas_pack_extended", _ptr(self.data), self.P, self.Ht, self.Wt, self.kind, _ptr(buf),
                     _stream())
                q = Filled(buf)
            self._quads = (q, version)
        q.use(stream)
        return q

    def pack(self, templates: torch.Tensor, st=None):
        """Fills the buffer from (P,Ht,Wt) f32 templates (extended atlases)."""
        self.fills += 1
        call("dbmp_atlas_pack_extended", _ptr(templates), self.P, self.Ht, self.Wt, self.kind, _ptr(self.data),
             st if st is not None else _stream())

    def private_copy(self, pixels: Optional[int] = None, N: int = 1 << 30) -> "Atlas":
        """An atlas of the same kind, templates and content bboxes with its own
        texel buffer (filled by the caller), for a job of N primitives on a canvas of
        `pixels` that re-derives its texels every step (the fit loop's blur
        schedule).  Such a job repacks an extended atlas every step, which an "f32"
        one only does where that pays."""
        a = Atlas.__new__(Atlas)
        a.templates, a.sigma, a.bbox = self.templates, self.sigma, self.bbox
        a.P, a.Ht, a.Wt, a.kind = self.P, self.Ht, self.Wt, self.kind
        a.extended = self.extended and (a.kind != ATLAS_F32 or pixels is None
                                        or quads_pay(pixels, N, self.templates.numel()))
        a.own, a._quads, a._anew, a._anew_next, a.fills = a.extended, None, 0, 0, 0
        if a.extended:
            a._alloc()
        else:
            a.data = torch.empty_like(self.templates)
        return a

    def with_kind(self, kind) -> "Atlas":
        a = Atlas(self.templates, kind)
        a.bbox, a.sigma = self.bbox, self.sigma   # keep the unblurred content bboxes
        return a


@dataclass
class TileLists:
    """CSR tile lists of one binning: offsets (T+1) and indices (>= L entries)."""
    offsets: torch.Tensor
    indices: torch.Tensor
    length: int

    def mapping_tensor(self) -> torch.Tensor:
        """The reference's int32 wire format [T+1, L, offsets..., indices...]."""
        head = torch.tensor([self.offsets.numel(), self.length], dtype=torch.int32, device=self.offsets.device)
        return torch.cat([head, self.offsets, self.indices[: self.length]])


@dataclass
class BatchState:
    """Forward state of a batch of candidates (Rasterizer.forward_batch):
    records (B*N,16), lists offsets (B,T+1) / indices (B,stride), per-pixel
    T_last / last_pos (B,H,W), the colour maps of a blended render."""
    prim_info: torch.Tensor
    offsets: torch.Tensor
    indices: torch.Tensor
    T_last: torch.Tensor
    last_pos: torch.Tensor
    colors_orig: Optional[torch.Tensor] = None
    cmap_stride: int = 0
    c_blend: float = 0.0
    walk_masks: Optional[torch.Tensor] = None    # what the forward's tests found (dbmp_render)
    atlas: Optional[Atlas] = None                # the forward's atlas
    quads: Optional[Filled] = None               # ... its packed copy, if the forward walked one
    fills: int = 0                               # ... and its fills

    @property
    def batch(self) -> int:
        return int(self.offsets.shape[0])


@dataclass
class ForwardState:
    prim_info: torch.Tensor
    lists: TileLists
    T_last: torch.Tensor
    last_pos: torch.Tensor
    colors_orig: Optional[torch.Tensor] = None   # colour maps of a blended render
    c_blend: float = 0.0
    walk_masks: Optional[torch.Tensor] = None    # what the forward's tests found (dbmp_render)
    atlas: Optional[Atlas] = None                # the forward's atlas
    quads: Optional[Filled] = None               # ... its packed copy, if the forward walked one
    fills: int = 0                               # ... and its fills


def lists_from_mapping(mapping: torch.Tensor, num_tiles: int, num_prims: int) -> TileLists:
    """Views a reference mapping tensor (simple_tile_renderer.py:757-766) as
    TileLists after validating it, so that no kernel can read outside it."""
    _need_cuda(mapping)
    m = mapping.to(torch.int32).contiguous()
    if m.dim() != 1 or m.numel() < num_tiles + 3:
        raise ValueError(f"tile mapping has {m.numel()} entries, need at least {num_tiles + 3}")
    offs = m[2:3 + num_tiles]
    idx = m[3 + num_tiles:]
    head = torch.stack([m[0], m[1], offs.min(), offs.max(), offs[-1]]).tolist()
    T1, L, omin, omax, olast = head
    if T1 != num_tiles + 1:
        raise ValueError(f"tile mapping is for {T1 - 1} tiles, canvas has {num_tiles}")
    if L != idx.numel() or olast != L or omin < 0 or omax > L:
        raise ValueError(f"inconsistent tile mapping (L={L}, indices={idx.numel()}, offsets in [{omin},{omax}], "
                         f"last offset {olast})")
    if idx.numel() == 0:
        idx = torch.zeros(1, dtype=torch.int32, device=m.device)
    return TileLists(offs, idx, int(L))


class Rasterizer:
    """One canvas.  Holds the binning capacity and scratch between calls."""

    def __init__(self, height: int, width: int, tile_size: int = 32, alpha_max: float = 1.0,
                 t_stop: float = DEFAULT_T_STOP, bin_mode: int = BIN_CONTENT, device=None):
        self.H, self.W, self.ts = int(height), int(width), int(tile_size)
        self.alpha_max = float(alpha_max)
        self.t_stop = float(t_stop)
        self.bin_mode = int(bin_mode)
        self.device = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
        self.tiles_x = (self.W + self.ts - 1) // self.ts
        self.tiles_y = (self.H + self.ts - 1) // self.ts
        self.T = self.tiles_x * self.tiles_y
        # a fit job's persistent lists and binning workspace (_ensure): one job, one
        # stream at a time
        self.capacity = 0
        self._ws = None
        self._idx = None
        # the renders allocate their lists and workspace per call, so that calls on
        # other streams or threads never share them; what they share is sizes, each
        # read and replaced in one step, and pinned buffers, each held by one call
        self._hint = None          # list capacity of the next render
        self._ws_need = (None, 0)  # workspace bytes of the last (batch, N)
        self._mask_bytes = None    # walk masks of one candidate
        self._pins = []            # pinned flag buffers not in use

    def __getstate__(self):
        # copies and pickles start without flag buffers: a copy of a pinned tensor is
        # not pinned, and the binning would write to an address the device does not have
        return {**self.__dict__, "_pins": []}

    def canvas(self, N: int, atlas: Atlas) -> Canvas:
        """The canvas of calls that pass atlas.data."""
        return Canvas(self.H, self.W, self.ts, int(N), atlas.P, atlas.Ht, atlas.Wt, atlas.kind, self.bin_mode,
                      self.alpha_max, self.t_stop, EXTENDED_ATLAS if atlas.own else 0)

    def _quads(self, atlas: Atlas, N: int, B: int, stream) -> Optional[Filled]:
        if atlas.own or not quads_pay(B * self.H * self.W, N, atlas.templates.numel()):
            return None
        return atlas.quads(stream)

    def walk_canvas(self, N: int, atlas: Atlas, quads: Optional[Filled], changed: int):
        """(canvas, atlas pointer) of a walk: on the packed copy `quads` of an "f32"
        atlas with its flags at `changed` (behind the records), or on atlas.data."""
        if quads is None:
            return self.canvas(N, atlas), _ptr(atlas.data)
        cv = FollowedCanvas(self.H, self.W, self.ts, int(N), atlas.P, atlas.Ht, atlas.Wt, atlas.kind, self.bin_mode,
                            self.alpha_max, self.t_stop, FOLLOWED_ATLAS, _ptr(atlas.data), changed)
        return cv, _ptr(quads.tensor)

    # -- binning -----------------------------------------------------------
    def _ensure(self, cv: Canvas, cap: int):
        if cap > self.capacity or self._ws is None:
            self.capacity = int(cap)
            self._idx = torch.empty(max(self.capacity, 1), dtype=torch.int32, device=self.device)
        nbytes = int(lib.dbmp_bin_workspace_bytes(ctypes.byref(cv), self.capacity))
        if self._ws is None or self._ws.numel() < nbytes + 256:
            self._ws = torch.empty(nbytes + 256, dtype=torch.uint8, device=self.device)

    def _ws_ptr(self):
        base = self._ws.data_ptr()
        return ctypes.c_void_p((base + 255) & ~255), self._ws.numel() - 256

    def _scratch(self, cv: Canvas, B: int, N: int, stream):
        """(tensor, workspace bytes): a binning's workspace, followed by two ints
        per candidate for its flags."""
        size, nbytes = self._ws_need     # read once: another thread may replace it
        if size != (B, N):
            need = int(lib.dbmp_bin_batch_workspace_bytes(ctypes.byref(cv), B))
            nbytes = (need + 255) & ~255
            self._ws_need = ((B, N), nbytes)
        if stream is None:
            return torch.empty(nbytes + 8 * B, dtype=torch.uint8, device=self.device), nbytes
        with torch.cuda.stream(stream):      # of the call's own stream, which frees it in its order
            return torch.empty(nbytes + 8 * B, dtype=torch.uint8, device=self.device), nbytes

    @staticmethod
    def _flat_batch(ts, stream):
        """The tensors contiguous: the batch calls step from candidate to candidate
        by N, but candidates may come strided or expanded.  Copied on the call's
        stream, on which the caller has them ready."""
        with _on(stream):
            return [t.contiguous() for t in ts]

    def _capacity(self, N: int) -> int:
        """List entries to provide per candidate: 1.25 times the longest lists so
        far, at first an eighth of all (tile, primitive) pairs up to 16 MB."""
        hint = self._hint
        if hint is None:
            self._hint = hint = min(N * self.T, max(N * self.T // 8, 1024) + 4096, 4 << 20)
        return hint

    def _grow_hint(self, L: int, indices: torch.Tensor, stream):
        """After a call on `stream` whose lists of up to L entries `indices` did not
        hold; the candidates that it did hold may still be walked there."""
        self._hint = min(max(self._hint, int(L * 1.25) + 4096), 0x7fffffff)
        if stream is not None:
            indices.record_stream(stream)

    def bin(self, means2D, radii, rotations, opacities, colors, sel, atlas: Atlas, stream=None):
        """Device binning.  Returns (prim_info, TileLists).  Synchronises once
        to learn the list length (the reference reads it with .item() too)."""
        N = int(radii.shape[0])
        cv = self.canvas(N, atlas)
        st = _stream(stream)
        prim_info = torch.empty((max(N, 1), 16), dtype=torch.float32, device=self.device)
        offsets = torch.empty(self.T + 1, dtype=torch.int32, device=self.device)
        ws, nbytes = self._scratch(cv, 1, N, stream)
        flags = ws[nbytes:nbytes + 8].view(torch.int32)
        for _ in range(3):
            # each binning owns its index list: a ForwardState must stay valid
            # while later forwards on this canvas run (batch APIs keep several)
            cap = self._capacity(N)
            indices = torch.empty(max(cap, 1), dtype=torch.int32, device=self.device)
            call("dbmp_bin", ctypes.byref(cv), _ptr(means2D), _ptr(radii), _ptr(rotations), _ptr(opacities),
                 _ptr(colors), _ptr(sel), _ptr(atlas.bbox), _ptr(prim_info), _ptr(offsets), _ptr(indices), cap,
                 _ptr(flags), flags.data_ptr() + 4, _ptr(ws), nbytes, st)
            with _on(stream):     # behind the binning
                L, overflow = flags.tolist()
            if not overflow:
                return prim_info, TileLists(offsets, indices, int(L))
            self._grow_hint(L, indices, stream)
        raise DbmpError("binning capacity did not converge")

    def _render(self, lead: tuple, means2D, radii, rotations, opacities, colors, sel, sel_stride: int, atlas: Atlas,
                stream, cmap=None, cmap_stride: int = 0, c_blend: float = 0.0, masks: bool = True):
        """Binning and forward of B candidates (lead: () for one, else (B,)) in one
        call; the host waits for the list lengths while the forward runs, and
        repeats the call if they exceed the capacity.  Returns (color, alpha,
        T_last, last_pos, prim_info, offsets, indices, longest list, walk_masks,
        the atlas's packed copy, its fills); masks: the render's backward will be wanted."""
        B = lead[0] if lead else 1
        N = int(radii.shape[-1])
        fills, quads = atlas.fills, None if atlas.own else self._quads(atlas, N, B, stream)
        dev, H, W = self.device, self.H, self.W
        color = torch.empty((*lead, H, W, 3), dtype=torch.float32, device=dev)
        alpha = torch.empty((*lead, H, W), dtype=torch.float32, device=dev)
        T_last = torch.empty((*lead, H, W), dtype=torch.float32, device=dev)
        last_pos = torch.empty((*lead, H, W), dtype=torch.int32, device=dev)
        prim = torch.empty((B * N + 1, 16), dtype=torch.float32, device=dev)     # (the last one: flags)
        cv, texels = self.walk_canvas(N, atlas, quads, prim.data_ptr() + 64 * B * N)
        offsets = torch.empty((*lead, self.T + 1), dtype=torch.int32, device=dev)
        walk = None
        if masks:
            if self._mask_bytes is None:
                self._mask_bytes = int(lib.dbmp_walk_mask_bytes(ctypes.byref(cv), 1))
            walk = torch.empty(self._mask_bytes * B, dtype=torch.uint8, device=dev)
        ws, nbytes = self._scratch(cv, B, N, stream)
        st = _stream(stream)
        try:
            pin = self._pins.pop()       # (one step: another thread may take the last one)
        except IndexError:
            pin = None
        if pin is None or pin.numel() < 2 * B:
            pin = torch.empty(2 * B, dtype=torch.int32).pin_memory()
        flags = pin.numpy()
        for _ in range(4):
            cap = self._capacity(N)
            stride = max(cap, 1)
            indices = torch.empty((*lead, stride), dtype=torch.int32, device=dev)
            call("dbmp_render", ctypes.byref(cv), B, _ptr(means2D), _ptr(radii), _ptr(rotations), _ptr(opacities),
                 _ptr(colors), _ptr(sel), sel_stride, _ptr(atlas.bbox), texels, _ptr(prim), _ptr(offsets),
                 _ptr(indices), stride, cap, ws.data_ptr() + nbytes, _ptr(pin), _ptr(cmap), cmap_stride,
                 float(c_blend) if cmap is not None else 0.0, _ptr(color), _ptr(alpha), _ptr(T_last), _ptr(last_pos),
                 _ptr(walk), _ptr(ws), nbytes, st)
            call("dbmp_render_wait", _ptr(pin), B, st)
            if quads is not None and flags[1] & 2:        # the copy is out of date: nothing was rendered
                atlas._missed()
                quads = None
                cv, texels = self.walk_canvas(N, atlas, None, 0)
                if stream is not None:
                    indices.record_stream(stream)
                continue
            if not flags[1:2 * B:2].any():
                L = int(flags[0:2 * B:2].max())
                self._pins.append(pin)
                return color, alpha, T_last, last_pos, prim, offsets, indices, L, walk, quads, fills
            self._grow_hint(int(flags[0:2 * B:2].max()), indices, stream)
        raise DbmpError("binning capacity did not converge")

    def prepare(self, means2D, radii, rotations, opacities, colors, sel, atlas: Atlas, stream=None,
                quads: Optional[Filled] = None):
        """The records of given lists' walk (of the packed copy `quads`: its flags are
        the last record)."""
        N = int(radii.shape[0])
        prim_info = torch.empty((N + 1 if quads is not None else max(N, 1), 16), dtype=torch.float32, device=self.device)
        cv, _ = self.walk_canvas(N, atlas, quads, prim_info.data_ptr() + 64 * N)
        call("dbmp_prepare", ctypes.byref(cv), _ptr(means2D), _ptr(radii), _ptr(rotations), _ptr(opacities),
             _ptr(colors), _ptr(sel), _ptr(prim_info), _stream(stream))
        return prim_info

    def _sums(self, grad_color, grad_alpha, rows: int, stream):
        """(colour, alpha gradients as operands, accumulator) of a backward, on its
        stream."""
        if stream is not None:
            with torch.cuda.stream(stream):
                return self._sums(grad_color, grad_alpha, rows, None)
        return (_operand(grad_color), _operand(grad_alpha) if grad_alpha is not None else None,
                torch.empty((max(rows, 1), 8), dtype=torch.float64, device=self.device))

    def _walk_of(self, state, N: int, rows: int, atlas: Atlas, stream):
        """(canvas, atlas pointer, masks pointer) of the backward of a forward's
        state: the forward's packed copy and masks where `atlas` is the forward's, and
        filled as it was then.  (Another one may hold anything, sharper or
        blurred templates, say: its backward tests again.)"""
        if state.atlas is not atlas or state.fills != atlas.fills:
            return self.canvas(N, atlas), _ptr(atlas.data), None
        if state.quads is None:
            return self.canvas(N, atlas), _ptr(atlas.data), _ptr(state.walk_masks)
        state.quads.use(stream)
        cv, texels = self.walk_canvas(N, atlas, state.quads, state.prim_info.data_ptr() + 64 * rows)
        return cv, texels, _ptr(state.walk_masks)

    # -- forward / backward -------------------------------------------------
    def forward(self, means2D, radii, rotations, opacities, colors, sel, atlas: Atlas,
                mapping: Optional[torch.Tensor] = None, stream=None, colors_orig: Optional[torch.Tensor] = None,
                c_blend: float = 0.0, for_backward: bool = True):
        """Returns (color (H,W,3), alpha (H,W), ForwardState).  for_backward: the
        state also keeps what speeds up its backward.  With
        colors_orig (N,Ht,Wt,3) and c_blend in (0, 1], fragment colours blend
        the per-primitive colour maps (dbmp_forward_blend)."""
        _need_cuda(means2D, radii, rotations, opacities, colors, sel)
        N = int(radii.shape[0])
        cmap = self._colour_maps(colors_orig, c_blend, N, atlas)
        if mapping is None or mapping.numel() == 0:
            color, alpha, T_last, last_pos, prim_info, offsets, indices, L, walk, quads, fills = self._render(
                (), means2D, radii, rotations, opacities, colors, sel, 0, atlas, stream, cmap, 0, c_blend, for_backward)
            return color, alpha, ForwardState(prim_info, TileLists(offsets, indices, L), T_last, last_pos, cmap,
                                              float(c_blend) if cmap is not None else 0.0, walk, atlas, quads, fills)
        lists = lists_from_mapping(mapping, self.T, N)
        quads = self._quads(atlas, N, 1, stream)
        prim_info = self.prepare(means2D, radii, rotations, opacities, colors, sel, atlas, stream, quads)
        cv, texels = self.walk_canvas(N, atlas, quads, prim_info.data_ptr() + 64 * N)
        color = torch.empty((self.H, self.W, 3), dtype=torch.float32, device=self.device)
        alpha = torch.empty((self.H, self.W), dtype=torch.float32, device=self.device)
        T_last = torch.empty((self.H, self.W), dtype=torch.float32, device=self.device)
        last_pos = torch.empty((self.H, self.W), dtype=torch.int32, device=self.device)
        if cmap is None:
            call("dbmp_forward", ctypes.byref(cv), _ptr(prim_info), texels, _ptr(lists.offsets),
                 _ptr(lists.indices), _ptr(color), _ptr(alpha), _ptr(T_last), _ptr(last_pos), _stream(stream))
            return color, alpha, ForwardState(prim_info, lists, T_last, last_pos, atlas=atlas, quads=quads)
        call("dbmp_forward_blend", ctypes.byref(cv), _ptr(prim_info), texels, _ptr(lists.offsets),
             _ptr(lists.indices), _ptr(cmap), ctypes.c_float(c_blend), _ptr(color), _ptr(alpha), _ptr(T_last),
             _ptr(last_pos), _stream(stream))
        return color, alpha, ForwardState(prim_info, lists, T_last, last_pos, cmap, float(c_blend), None, atlas, quads)

    # -- batches of candidates -------------------------------------------------
    def bin_batch(self, means2D, radii, rotations, opacities, colors, sel, atlas: Atlas, stream=None):
        """Device binning of B candidates (leading dimension of every parameter
        tensor; sel (N) shared or (B,N)) into slots of shared buffers: records
        (B*N,16), offsets (B,T+1), indices (B,capacity).  One host
        synchronisation reads the B list lengths."""
        B, N = int(radii.shape[0]), int(radii.shape[1])
        cv = self.canvas(N, atlas)
        st = _stream(stream)
        prim = torch.empty((max(B * N, 1), 16), dtype=torch.float32, device=self.device)
        offsets = torch.empty((B, self.T + 1), dtype=torch.int32, device=self.device)
        small = torch.empty((B, 2), dtype=torch.int32, device=self.device)    # per candidate: L, overflow
        sel_stride = N if sel.dim() == 2 else 0
        if B == 0:
            return prim, offsets, torch.empty((0, 1), dtype=torch.int32, device=self.device)
        means2D, radii, rotations, opacities, colors, sel = self._flat_batch(
            (means2D, radii, rotations, opacities, colors, sel), stream)
        n = min(B, 65535)                       # candidates of one call
        ws, nbytes = self._scratch(cv, n, N, stream)
        for _ in range(3):
            cap = self._capacity(N)
            stride = max(cap, 1)
            indices = torch.empty((B, stride), dtype=torch.int32, device=self.device)
            for b in range(0, B, n):
                call("dbmp_bin_batch", ctypes.byref(cv), min(n, B - b), _ptr(means2D[b]), _ptr(radii[b]),
                     _ptr(rotations[b]), _ptr(opacities[b]), _ptr(colors[b]),
                     _ptr(sel[b]) if sel_stride else _ptr(sel), sel_stride, _ptr(atlas.bbox),
                     prim.data_ptr() + b * N * 64, _ptr(offsets[b]), _ptr(indices[b]), stride, cap, _ptr(small[b]),
                     _ptr(ws), nbytes, st)
            with _on(stream):     # behind the binning
                Ls = small.cpu()
            if not bool(Ls[:, 1].any()):
                return prim, offsets, indices
            self._grow_hint(int(Ls[:, 0].max()), indices, stream)
        raise DbmpError("binning capacity did not converge")

    def forward_batch(self, means2D, radii, rotations, opacities, colors, sel, atlas: Atlas, mappings=None,
                      stream=None, colors_orig: Optional[torch.Tensor] = None, c_blend: float = 0.0,
                      for_backward: bool = True):
        """B candidates of this canvas in one launch.  means2D (B,N,2), radii /
        rotations / opacities (B,N), colors (B,N,3), sel (N) or (B,N);
        mappings: None (device binning) or B reference mapping tensors;
        colors_orig (N,Ht,Wt,3) shared or (B,N,Ht,Wt,3).  Returns
        (color (B,H,W,3), alpha (B,H,W), BatchState)."""
        _need_cuda(means2D, radii, rotations, opacities, colors, sel)
        B, N = int(radii.shape[0]), int(radii.shape[1])
        st = _stream(stream)
        cmap, cstride = None, 0
        if colors_orig is not None and colors_orig.numel() > 0 and float(c_blend) > 0.0:
            if colors_orig.dim() == 5:
                cmap = self._colour_maps(colors_orig.reshape(B * N, *colors_orig.shape[2:]), c_blend, B * N, atlas)
                cstride = N * atlas.Ht * atlas.Wt * 3
            else:
                cmap = self._colour_maps(colors_orig, c_blend, N, atlas)
        has_maps = mappings is not None and len(mappings) > 0
        if not has_maps and 0 < B <= 65535:
            params = self._flat_batch((means2D, radii, rotations, opacities, colors, sel), stream)
            color, alpha, T_last, last_pos, prim, offsets, indices, _, walk, quads, fills = self._render(
                (B,), *params, N if sel.dim() == 2 else 0, atlas, stream, cmap, cstride, c_blend, for_backward)
            return color, alpha, BatchState(prim, offsets, indices, T_last, last_pos, cmap, cstride,
                                            float(c_blend) if cmap is not None else 0.0, walk, atlas, quads, fills)
        quads = None
        if has_maps:
            quads = self._quads(atlas, N, B, stream)
            if len(mappings) != B:
                raise ValueError(f"{len(mappings)} mappings for {B} candidates")
            lists = [lists_from_mapping(m, self.T, N) for m in mappings]
            stride = max(max(l.length for l in lists), 1)
            offsets = torch.stack([l.offsets for l in lists])
            indices = torch.zeros((B, stride), dtype=torch.int32, device=self.device)
            for b, l in enumerate(lists):
                indices[b, :l.length] = l.indices[:l.length]
            prim = torch.empty((B * N + 1, 16), dtype=torch.float32, device=self.device)    # (the last one: flags)
            cv, _ = self.walk_canvas(N, atlas, quads, prim.data_ptr() + 64 * B * N)
            sel2 = sel if sel.dim() == 2 else sel.unsqueeze(0).expand(B, -1)
            for b in range(B):
                call("dbmp_prepare", ctypes.byref(cv), _ptr(means2D[b]), _ptr(radii[b]), _ptr(rotations[b]),
                     _ptr(opacities[b]), _ptr(colors[b]), _ptr(sel2[b]),
                     ctypes.c_void_p(prim.data_ptr() + b * N * 64), st)
        else:
            prim, offsets, indices = self.bin_batch(means2D, radii, rotations, opacities, colors, sel, atlas, stream)
        cv, texels = self.walk_canvas(N, atlas, quads, prim.data_ptr() + 64 * B * N)
        dev = self.device
        color = torch.empty((B, self.H, self.W, 3), dtype=torch.float32, device=dev)
        alpha = torch.empty((B, self.H, self.W), dtype=torch.float32, device=dev)
        T_last = torch.empty((B, self.H, self.W), dtype=torch.float32, device=dev)
        last_pos = torch.empty((B, self.H, self.W), dtype=torch.int32, device=dev)
        call("dbmp_forward_batch", ctypes.byref(cv), B, _ptr(prim), texels, _ptr(offsets), _ptr(indices),
             ctypes.c_longlong(indices.shape[1]), _ptr(cmap), ctypes.c_longlong(cstride),
             ctypes.c_float(c_blend if cmap is not None else 0.0), _ptr(color), _ptr(alpha), _ptr(T_last),
             _ptr(last_pos), st)
        return color, alpha, BatchState(prim, offsets, indices, T_last, last_pos, cmap, cstride,
                                        float(c_blend) if cmap is not None else 0.0, None, atlas, quads)

    def backward_batch(self, state: BatchState, grad_color, grad_alpha, radii, rotations, opacities, colors,
                       atlas: Atlas, stream=None):
        """The five gradients of each candidate, in one launch: (B,N,2),
        (B,N), (B,N), (B,N), (B,N,3)."""
        B, N = int(radii.shape[0]), int(radii.shape[1])
        dev = self.device
        gc, ga, acc = self._sums(grad_color, grad_alpha, B * N, stream)
        cv, texels, masks = self._walk_of(state, N, B * N, atlas, stream)
        outs = [torch.empty(sh, dtype=torch.float32, device=dev)
                for sh in ((B, N, 2), (B, N), (B, N), (B, N), (B, N, 3))]
        call("dbmp_backward_masked", ctypes.byref(cv), B, masks, _ptr(state.prim_info),
             texels, _ptr(state.offsets), _ptr(state.indices), state.indices.shape[1],
             _ptr(state.colors_orig), state.cmap_stride, float(state.c_blend),
             _ptr(state.T_last), _ptr(state.last_pos), _ptr(gc), _ptr(ga), _ptr(radii), _ptr(rotations),
             _ptr(opacities), _ptr(colors), _ptr(acc), *[_ptr(o) for o in outs], _stream(stream))
        return tuple(outs)

    @staticmethod
    def _colour_maps(colors_orig, c_blend, N, atlas: Atlas):
        """The (N,Ht,Wt,3) f32 colour maps of a blended render, or None."""
        if colors_orig is None or colors_orig.numel() == 0 or float(c_blend) <= 0.0:
            return None
        if not 0.0 < float(c_blend) <= 1.0:
            raise ValueError(f"c_blend {c_blend} outside [0, 1]")
        _need_cuda(colors_orig)
        cm = _f32(colors_orig)
        if cm.numel() != N * atlas.Ht * atlas.Wt * 3:
            raise ValueError(f"colors_orig has {cm.numel()} values, expected N*Ht*Wt*3 = "
                             f"{N}*{atlas.Ht}*{atlas.Wt}*3")
        return cm

    def backward(self, state: ForwardState, grad_color, grad_alpha, radii, rotations, opacities, colors,
                 atlas: Atlas, stream=None):
        """Returns the reference's five gradients: (means2D (N,2), radii (N),
        rotations (N), opacities (N), colors (N,3)), float32."""
        N = int(radii.shape[0])
        dev = self.device
        gc, ga, acc = self._sums(grad_color, grad_alpha, N, stream)
        cv, texels, masks = self._walk_of(state, N, N, atlas, stream)
        g_means = torch.empty((N, 2), dtype=torch.float32, device=dev)
        g_r = torch.empty(N, dtype=torch.float32, device=dev)
        g_rot = torch.empty(N, dtype=torch.float32, device=dev)
        g_op = torch.empty(N, dtype=torch.float32, device=dev)
        g_col = torch.empty((N, 3), dtype=torch.float32, device=dev)
        call("dbmp_backward_masked", ctypes.byref(cv), 1, masks, _ptr(state.prim_info),
             texels, _ptr(state.lists.offsets), _ptr(state.lists.indices), state.lists.indices.numel(),
             _ptr(state.colors_orig), 0, float(state.c_blend) if state.colors_orig is not None else 0.0,
             _ptr(state.T_last), _ptr(state.last_pos), _ptr(gc), _ptr(ga), _ptr(radii), _ptr(rotations),
             _ptr(opacities), _ptr(colors), _ptr(acc), _ptr(g_means), _ptr(g_r), _ptr(g_rot), _ptr(g_op), _ptr(g_col),
             _stream(stream))
        return g_means, g_r, g_rot, g_op, g_col


def _flat(t: torch.Tensor) -> torch.Tensor:
    return t if t.dim() == 1 else t.view(-1)


def _shaped(t: torch.Tensor, k: int) -> torch.Tensor:
    return t if t.dim() == 2 and t.shape[1] == k else t.view(-1, k)


class RasterizeFunction(torch.autograd.Function):
    """Differentiable render of bitmap primitives (hand-written backward).

    forward(means2D (N,2), radii (N), rotations (N), opacities (N), colors (N,3),
            sel (N) int, atlas, rasterizer, mapping, colors_orig, c_blend)
        -> (color (H,W,3), alpha (H,W))
    Gradients flow to the five parameter tensors, as in the reference's
    TileRasterizerFunction (cuda_tile_rasterizer/__init__.py:254-340); the
    colour maps colors_orig get none, as there.
    """

    @staticmethod
    def forward(ctx, means2D, radii, rotations, opacities, colors, sel, atlas, rasterizer, mapping=None,
                colors_orig=None, c_blend=0.0):
        m, r, th, v, c = (_operand(t) for t in (means2D, radii, rotations, opacities, colors))
        s = sel.detach().to(torch.int32).contiguous()
        color, alpha, state = rasterizer.forward(_shaped(m, 2), _flat(r), _flat(th), _flat(v), _shaped(c, 3),
                                                 _flat(s), atlas, mapping, None,
                                                 None if colors_orig is None else colors_orig.detach(),
                                                 float(c_blend), any(ctx.needs_input_grad[:5]))
        ctx.state = state
        ctx.atlas = atlas
        ctx.rasterizer = rasterizer
        ctx.shapes = (means2D.shape, radii.shape, rotations.shape, opacities.shape, colors.shape)
        ctx.save_for_backward(r, th, v, c)
        return color, alpha

    @staticmethod
    def backward(ctx, grad_color, grad_alpha):
        r, th, v, c = ctx.saved_tensors
        rz: Rasterizer = ctx.rasterizer
        if grad_color is None:
            grad_color = torch.zeros((rz.H, rz.W, 3), dtype=torch.float32, device=r.device)
        g = rz.backward(ctx.state, grad_color, grad_alpha, _flat(r), _flat(th), _flat(v), _shaped(c, 3), ctx.atlas)
        return (*(x if x.shape == sh else x.view(sh) for x, sh in zip(g, ctx.shapes)),
                None, None, None, None, None, None)


class RasterizeBatchFunction(torch.autograd.Function):
    """Differentiable render of B candidates in one launch per direction.

    forward(means2D (B,N,2), radii (B,N), rotations (B,N), opacities (B,N),
            colors (B,N,3), sel (N) or (B,N), atlas, rasterizer, mappings,
            colors_orig, c_blend) -> (color (B,H,W,3), alpha (B,H,W))
    Gradients flow to the five parameter tensors of every candidate, as in the
    reference's TileRasterizerBatchFunction (cuda_tile_rasterizer/__init__.py:
    124-252), whose backward loops over the candidates.
    """

    @staticmethod
    def forward(ctx, means2D, radii, rotations, opacities, colors, sel, atlas, rasterizer, mappings=None,
                colors_orig=None, c_blend=0.0):
        B = int(radii.shape[0])
        m, r, th, v, c = (_operand(t) for t in (means2D, radii, rotations, opacities, colors))
        s = sel.detach().to(torch.int32).contiguous()
        color, alpha, state = rasterizer.forward_batch(m.view(B, -1, 2), r.view(B, -1), th.view(B, -1),
                                                       v.view(B, -1), c.view(B, -1, 3), s, atlas, mappings, None,
                                                       None if colors_orig is None else colors_orig.detach(),
                                                       float(c_blend), any(ctx.needs_input_grad[:5]))
        ctx.state, ctx.atlas, ctx.rasterizer = state, atlas, rasterizer
        ctx.shapes = (means2D.shape, radii.shape, rotations.shape, opacities.shape, colors.shape)
        ctx.save_for_backward(r, th, v, c)
        return color, alpha

    @staticmethod
    def backward(ctx, grad_color, grad_alpha):
        r, th, v, c = ctx.saved_tensors
        rz: Rasterizer = ctx.rasterizer
        B = int(ctx.state.batch)
        if grad_color is None:
            grad_color = torch.zeros((B, rz.H, rz.W, 3), dtype=torch.float32, device=r.device)
        g = rz.backward_batch(ctx.state, grad_color, grad_alpha, r.view(B, -1), th.view(B, -1), v.view(B, -1),
                              c.view(B, -1, 3), ctx.atlas)
        sh = ctx.shapes
        return (g[0].view(sh[0]), g[1].view(sh[1]), g[2].view(sh[2]), g[3].view(sh[3]), g[4].view(sh[4]),
                None, None, None, None, None, None)


def rasterize_batch(means2D, radii, rotations, opacities, colors, sel, atlas: Atlas, rasterizer: Rasterizer,
                    mappings=None, colors_orig: Optional[torch.Tensor] = None, c_blend: float = 0.0):
    return RasterizeBatchFunction.apply(means2D, radii, rotations, opacities, colors, sel, atlas, rasterizer,
                                        mappings, colors_orig, c_blend)


def rasterize(means2D, radii, rotations, opacities, colors, sel, atlas: Atlas, rasterizer: Rasterizer,
              mapping: Optional[torch.Tensor] = None, colors_orig: Optional[torch.Tensor] = None,
              c_blend: float = 0.0):
    return RasterizeFunction.apply(means2D, radii, rotations, opacities, colors, sel, atlas, rasterizer, mapping,
                                   colors_orig, c_blend)
