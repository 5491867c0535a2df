"""Shared implementation of the drop-in extension modules `_C` and `_C_fp16`.

The reference's extensions (cuda_tile_rasterizer/ext.cpp:5-121 and
ext_fp16.cpp:5-83) keep one process-global TileRasterizer that owns the
per-pixel caches between a forward and the following backward.  This module
keeps the same global-by-design contract (init_* replaces it) on top of
libdbmp.so: the forward keeps its ForwardState, the backward consumes it.
Every computation runs in the library's CUDA kernels; there is no fallback.
"""
from __future__ import annotations

import ctypes
import time

import torch

from diffbmp_b200 import rasterizer as R


class _Global:
    def __init__(self, H, W, ts, alpha_ub, fp16):
        self.H, self.W, self.ts = int(H), int(W), int(ts)
        self.alpha_ub = float(alpha_ub)
        self.fp16 = fp16
        self.kind = "f16" if fp16 else "f32"
        # an empty mapping means "every primitive in every tile" in the reference
        # (tile_rasterize.cu:171-194); the cull-square binning is its tight form
        self.rz_cull = R.Rasterizer(H, W, ts, alpha_ub, bin_mode=R.BIN_CULL)
        self.rz_map = R.Rasterizer(H, W, ts, alpha_ub, bin_mode=R.BIN_CONTENT)
        self.atlas_key = None
        self.atlas = None
        self.atlas_templates = None    # the keyed tensor: alive, so that no other one gets its address
        self.states = []
        self.batch_state = None     # (BatchState, rasterizer, atlas) of the last forward_batch
        self.t_fwd = self.t_bwd = 0.0
        self.n_fwd = self.n_bwd = 0

    def get_atlas(self, templates: torch.Tensor) -> R.Atlas:
        t = templates if templates.dim() == 3 else templates.unsqueeze(0)
        key = (t.data_ptr(), tuple(t.shape), t.stride(), t._version, t.dtype)
        if key != self.atlas_key:
            self.atlas = R.Atlas(t.float(), self.kind)
            self.atlas_key, self.atlas_templates = key, t.detach()
        return self.atlas


_G: dict = {}


def init(H, W, ts, sigma, alpha_ub, max_prims_per_pixel, num_primitives, fp16=False):
    """init_tile_rasterizer(H, W, tile_size, sigma, alpha_upper_bound,
    max_prims_per_pixel, num_primitives): max_prims_per_pixel is accepted and
    unused (no per-layer caches exist here, depth is unbounded)."""
    _G[fp16] = _Global(H, W, ts, alpha_ub, fp16)


def _get(fp16):
    g = _G.get(fp16)
    if g is None:
        raise RuntimeError("TileRasterizer not initialized. Call init_tile_rasterizer first.")
    return g


def _f(t):
    return t.detach().to(torch.float32).contiguous()


def _convert(ts, dtype):
    """Contiguous CUDA tensors of one device and one dtype to the other of float16
    / float32, in one launch per eight."""
    out = [torch.empty(t.shape, dtype=dtype, device=t.device) for t in ts]
    for k in range(0, len(ts), 8):
        a, b = ts[k:k + 8], out[k:k + 8]
        n = len(a)
        R.call("dbmp_convert_half", n, (ctypes.c_void_p * n)(*[t.data_ptr() for t in a]),
               (ctypes.c_void_p * n)(*[t.data_ptr() for t in b]), (ctypes.c_longlong * n)(*[t.numel() for t in a]),
               int(dtype is torch.float16), R._stream())
    return out


def _floats(*ts):
    """Each tensor (or None) as contiguous f32, the half ones converted together."""
    out = [t if t is None else t.detach() for t in ts]
    todo = [k for k, t in enumerate(out) if t is not None and t.dtype is torch.float16 and t.is_cuda
            and t.is_contiguous()]
    for k, t in zip(todo, _convert([out[k] for k in todo], torch.float32)):
        out[k] = t
    return [t if t is None else R._operand(t) for t in out]


def _halves(ts):
    return tuple(_convert([t.contiguous() for t in ts], torch.float16))


def forward(fp16, means2D, radii, rotations, opacities, colors, colors_orig, templates, sel, c_blend, mapping,
            keep=True):
    g = _get(fp16)
    t0 = time.perf_counter()
    atlas = g.get_atlas(templates)
    m, r, th, v, c = _floats(means2D, radii, rotations, opacities, colors)
    m, r, th, v, c = m.view(-1, 2), r.view(-1), th.view(-1), v.view(-1), c.view(-1, 3)
    s = sel.to(torch.int32).contiguous().view(-1)
    has_map = mapping is not None and isinstance(mapping, torch.Tensor) and mapping.numel() > 0
    rz = g.rz_map if has_map else g.rz_cull
    # colour-map blending (tile_forward.cu:316-330) when colors_orig is given and c_blend > 0
    blend = colors_orig is not None and isinstance(colors_orig, torch.Tensor) and colors_orig.numel() > 0 \
        and float(c_blend) > 0.0
    color, alpha, state = rz.forward(m, r, th, v, c, s, atlas, mapping if has_map else None, None,
                                     _f(colors_orig) if blend else None, float(c_blend) if blend else 0.0)
    if keep:
        g.states = [(state, rz, atlas)]
    g.t_fwd += (time.perf_counter() - t0) * 1e3
    g.n_fwd += 1
    if fp16:
        return _halves((color, alpha))
    return color, alpha, (state, rz, atlas)


def backward(fp16, grad_color, grad_alpha, radii, rotations, opacities, colors, saved=None):
    g = _get(fp16)
    if saved is None:
        if not g.states:
            raise RuntimeError("TileRasterizer not initialized or forward pass not called.")
        saved = g.states[-1]
    state, rz, atlas = saved
    t0 = time.perf_counter()
    gcol, galp, r, th, v, c = _floats(grad_color, grad_alpha, radii, rotations, opacities, colors)
    out = rz.backward(state, gcol, galp, r.view(-1), th.view(-1), v.view(-1), c.view(-1, 3), atlas)
    if fp16:
        out = _halves(out)
    g.t_bwd += (time.perf_counter() - t0) * 1e3
    g.n_bwd += 1
    return out


def forward_batch(fp16, means2D, radii, rotations, opacities, colors, colors_orig, templates, sel, c_blend,
                  mappings):
    """B candidates (leading dimension) in one forward launch.  mappings: a
    list of B reference mapping tensors, one tensor shared by every candidate
    (the FP16 extension's form, tile_rasterize_fp16.cpp:501-560), or None
    (device binning per candidate).  Keeps the batch state for backward_batch
    and returns (color (B,H,W,3), alpha (B,H,W))."""
    g = _get(fp16)
    t0 = time.perf_counter()
    atlas = g.get_atlas(templates)
    B = int(radii.shape[0])
    m, r, th, v, c = _floats(means2D, radii, rotations, opacities, colors)
    m, r, th, v, c = m.view(B, -1, 2), r.view(B, -1), th.view(B, -1), v.view(B, -1), c.view(B, -1, 3)
    s = sel.to(torch.int32).contiguous()
    if isinstance(mappings, torch.Tensor):
        mappings = [mappings] * B if mappings.numel() > 0 else None
    elif mappings is not None:
        mappings = [mp for mp in mappings if mp is not None and mp.numel() > 0] or None
    rz = g.rz_map if mappings is not None else g.rz_cull
    blend = colors_orig is not None and isinstance(colors_orig, torch.Tensor) and colors_orig.numel() > 0 \
        and float(c_blend) > 0.0
    color, alpha, state = rz.forward_batch(m, r, th, v, c, s, atlas, mappings, None,
                                           _f(colors_orig) if blend else None, float(c_blend) if blend else 0.0)
    g.batch_state = (state, rz, atlas)
    g.t_fwd += (time.perf_counter() - t0) * 1e3
    g.n_fwd += 1
    if fp16:
        return _halves((color, alpha))
    return color, alpha


def backward_batch(fp16, grad_color, grad_alpha, radii, rotations, opacities, colors):
    """The five gradients of every candidate of the last forward_batch, one
    backward launch: (B,N,2), (B,N), (B,N), (B,N), (B,N,3)."""
    g = _get(fp16)
    if getattr(g, "batch_state", None) is None:
        raise RuntimeError("backward_batch must follow a forward_batch")
    state, rz, atlas = g.batch_state
    B = int(radii.shape[0])
    if state.batch != B:
        raise RuntimeError(f"backward_batch of {B} candidates after a forward_batch of {state.batch}")
    t0 = time.perf_counter()
    gcol, galp, r, th, v, c = _floats(grad_color, grad_alpha, radii, rotations, opacities, colors)
    out = rz.backward_batch(state, gcol, galp, r.view(B, -1), th.view(B, -1), v.view(B, -1), c.view(B, -1, 3), atlas)
    if fp16:
        out = _halves(out)
    g.t_bwd += (time.perf_counter() - t0) * 1e3
    g.n_bwd += 1
    return out


def timing_stats(fp16):
    g = _G.get(fp16)
    if g is None:
        print("No TileRasterizer instance available for timing stats.")
        return
    print("=== CUDA Tile Rasterizer Timing Statistics ===")
    print(f"Forward Pass: total {g.t_fwd:.3f} ms over {g.n_fwd} iterations (host wall time, asynchronous launches)")
    print(f"Backward Pass: total {g.t_bwd:.3f} ms over {g.n_bwd} iterations")


def reset_timing(fp16):
    g = _G.get(fp16)
    if g is not None:
        g.t_fwd = g.t_bwd = 0.0
        g.n_fwd = g.n_bwd = 0
    print("Timing statistics reset.")
