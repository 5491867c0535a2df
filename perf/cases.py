"""Timed cases of the rasterizer: the calls that a user's program makes, over the sizes it makes them at.

Canvases, primitive counts, atlases and parameter distributions are those of diffbmp_b200.workloads, of the tests and
of bench.py (64x64 with 32 primitives up to 4096x4096 with 100,000), with ragged sizes in between.  A case is one of
six operations ("op"):

  render  SimpleTileRenderer.render_from_params without gradients: a preview or the final image over a background
  grad    rasterize() and its backward with a given image gradient: one step of a program with a loss of its own
  dropin  the reference's TileRasterizer object and its backward, FP16 tensors in and out
  batch   rasterize_batch() of B candidates and its backward
  fit     one iteration of a resident ImageFitter (binning, fused kernel, Adam) on freshly uploaded parameters
  loop    SimpleTileRenderer.optimize_parameters: a whole short fit with decay, blur schedule and pruning
  psd     the layer crops of a PSD export and their PackBits channel blocks
"""
import math

import numpy as np
import torch

from diffbmp_b200 import cuda_tile_rasterizer as ctr
from diffbmp_b200 import psd
from diffbmp_b200 import workloads as wl
from diffbmp_b200.fitting import FitConfig, ImageFitter
from diffbmp_b200.pydiffbmp.core.renderer.simple_tile_renderer import SimpleTileRenderer
from diffbmp_b200.rasterizer import Atlas, Rasterizer, rasterize, rasterize_batch


def _case(name, op, H, W, N, P, th, tw, **more):
    return dict(dict(name=name, op=op, H=H, W=W, N=N, P=P, th=th, tw=tw, kind="f32", tile=32, alpha_max=1.0), **more)


def listed():
    return [
        # the gradient-check scene: the smallest call, all launches and host work
        _case("grad_64", "grad", 64, 64, 32, 1, 32, 32),
        # an interactive preview of a small job, no gradients, the renderer API's default opacity bound
        _case("render_256", "render", 256, 256, 512, 1, 64, 64, alpha_max=0.5),
        # an existing caller of the reference's FP16 extension: its default tile size 16, ragged canvas
        _case("dropin_f16_333x500", "dropin", 333, 500, 700, 3, 64, 64, kind="f16", tile=16),
        # primitives with their own colour maps (c_blend), a photo-mosaic job
        _case("grad_cmap_512", "grad", 512, 512, 300, 4, 64, 64, c_blend=0.4),
        # four candidate parameter sets of one canvas, ranked by a caller's own loss
        _case("batch4_384x512", "batch", 384, 512, 800, 4, 96, 96, kind="f16q", B=4),
        # one iteration of a small serving job in the precision form
        _case("fit_f16q_256x512", "fit", 256, 512, 700, 16, 256, 256, kind="f16q"),
        # a whole short fit as the reference's config drives it: decay, adaptive blur, pruning, FP32
        _case("loop_512", "loop", 512, 512, 600, 8, 128, 128, iters=5),
        # odd sizes, non-square bitmaps, bfloat16 storage, a bounded opacity
        _case("grad_bf16_717x1301", "grad", 717, 1301, 2500, 5, 121, 90, kind="bf16", alpha_max=0.8),
        # the mid-size workload in plain FP32: one training step of a program with its own loss
        _case("grad_1024", "grad", 1024, 1024, 5000, 8, 128, 128),
        # a layered export of a mid-size result
        _case("psd_1024", "psd", 1024, 1024, 1500, 8, 128, 128),
        # the headline workload: one fit iteration, FP16 storage, parameters from the host
        _case("fit_f16q_2048", "fit", 2048, 2048, 20000, 16, 256, 256, kind="f16q"),
        # the deep scene: 4096x4096, thousands of layers per pixel
        _case("grad_4096", "grad", 4096, 4096, 100000, 1, 64, 64),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["grad", "grad", "grad", "fit", "fit", "fit", "render", "batch", "dropin", "cmap", "loop", "psd"])
    kinds = ["f32", "f32", "f16q", "f16", "bf16q", "bf16"]
    th = _between(rng, 24, 256)
    tw = th if rng.random() < 0.7 else _between(rng, 24, 256)
    P = _between(rng, 1, 16)
    c = dict(op=op, P=P, th=th, tw=tw, kind=rng.choice(kinds), tile=32, alpha_max=rng.choice([1.0, 1.0, 0.8, 0.5]))
    if op == "render":
        c.update(H=_between(rng, 64, 2048), W=_between(rng, 64, 2048), N=_between(rng, 32, 20000),
                 kind=rng.choice(["f32", "f16q"]))
    elif op == "dropin":
        c.update(H=_between(rng, 64, 768), W=_between(rng, 64, 768), N=_between(rng, 32, 2000), kind="f16",
                 tile=rng.choice([16, 32]), alpha_max=1.0)
    elif op == "cmap":
        c.update(op="grad", H=_between(rng, 64, 768), W=_between(rng, 64, 768), N=_between(rng, 16, 600),
                 c_blend=rng.choice([0.2, 0.5, 1.0]))
    elif op == "batch":
        c.update(H=_between(rng, 64, 768), W=_between(rng, 64, 768), N=_between(rng, 32, 2000), B=rng.randint(2, 8))
    elif op == "loop":
        c.update(H=_between(rng, 128, 768), W=_between(rng, 128, 768), N=_between(rng, 64, 1000), iters=5, P=max(P, 2),
                 kind=rng.choice(["f32", "f16q"]))
    elif op == "psd":
        c.update(H=_between(rng, 128, 1400), W=_between(rng, 128, 1400), N=_between(rng, 32, 2000), kind="f32")
    elif op == "fit":
        c.update(H=_between(rng, 128, 2048), W=_between(rng, 128, 2048), N=_between(rng, 128, 20000))
    else:
        c.update(H=_between(rng, 64, 2048), W=_between(rng, 64, 2048), N=_between(rng, 32, 20000),
                 tile=32 if rng.random() < 0.8 else 16)
    return c


# ---------------------------------------------------------------------------
# Inputs
def _shape(rng, s, turns):
    """A random soft shape; with turns, one that a rotation changes (no ring)."""
    t = wl.random_shape(rng, s)
    while turns and np.abs(t - t.T).mean() < 0.01:
        t = wl.random_shape(rng, s)
    return t


def _templates(rng, op, P, th, tw):
    """P soft shapes, cropped around the centre when th != tw: a disk for a render of one bitmap.  Gradients of a lone
    bitmap and fits of several steps take shapes that a rotation changes: the rotation gradient of others is rounding
    alone, and Adam scales that to full steps."""
    s = max(th, tw)
    turns = op == "loop" or P == 1
    t = np.stack([wl.soft_disk(s, 0.375 * s) if P == 1 and op == "render" else _shape(rng, s, turns) for _ in range(P)])
    y, x = (s - th) // 2, (s - tw) // 2
    return np.ascontiguousarray(t[:, y:y + th, x:x + tw])


def _inputs(case, seed):
    """Host arrays of a case: templates and B parameter sets (B = 1 outside batches)."""
    rng = np.random.default_rng(seed)
    H, W, N, P = case["H"], case["W"], case["N"], case["P"]
    api = case["op"] in ("render", "loop")     # the renderer API assigns template (N-1-i) % P itself
    t = _templates(rng, case["op"], P, case["th"], case["tw"])
    sets = [list(wl.sample_params(rng, H, W, N, P, "reference" if api else "uniform")) for _ in range(case.get("B", 1))]
    for s in sets:
        s[5] = sets[0][5]
        if case["op"] == "psd":
            s[1] = s[1] * np.float32(0.5)
        if case["op"] == "dropin":             # half tensors carry the parameters
            s[:5] = [a.astype(np.float16) for a in s[:5]]
            s[0], s[1] = np.clip(s[0], 0, 2000), np.clip(s[1], 0, 2000)
    if case["op"] == "dropin":
        t = t.astype(np.float16)
    return rng, t, sets


def _dev(a, dtype=None):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


def _upstream(case, seed):
    """The image gradients of the caller's loss."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    shape = (case["H"], case["W"]) if case["op"] != "batch" else (case["B"], case["H"], case["W"])
    return (torch.randn(*shape, 3, generator=g, device="cuda"), torch.randn(*shape, generator=g, device="cuda"))


def _target(case, seed):
    return wl.smooth_field_device(np.random.default_rng(seed + 5), case["H"], case["W"], "cuda", noise=0.02)


def _loop_conf(case):
    return dict(num_iterations=case["iters"], learning_rate=dict(default=0.01), do_decay=True, decay_rate=0.99,
                do_adapt_gaussian_blur=True, blur_sigma_start=2.0, blur_sigma_end=0.0, bg_color="white",
                pruning=dict(do_pruning=True, prune_threshold=0.3, prune_iterations=3, no_prune_last_iterations=1,
                             no_prune_warmup_iterations=1))


class _Pool:
    """The caller's initializer: replacement primitives for pruning."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed

    def reinitialize_subset(self, rows, target, device):
        g = torch.Generator(device="cuda").manual_seed(self.seed + 13)
        u = torch.rand(rows, 8, generator=g, device="cuda")
        H, W = self.case["H"], self.case["W"]
        return (u[:, 0] * W, u[:, 1] * H, u[:, 2] * (min(H, W) / 20) + 2, torch.full_like(u[:, 0], -2.0),
                u[:, 3] * 6.28, u[:, 5:8])


def prepare(case, seed):
    rng, t, sets = _inputs(case, seed)
    H, W, op = case["H"], case["W"], case["op"]
    s = dict(case=case, op=op)
    p = [_dev(np.stack([q[k] for q in sets]) if op == "batch" else sets[0][k]) for k in range(5)]
    s["sel"] = _dev(sets[0][5])
    tmpl = _dev(t)
    if op in ("render", "loop"):
        s["renderer"] = SimpleTileRenderer((H, W), tmpl, tile_size=case["tile"], alpha_upper_bound=case["alpha_max"],
                                           use_fp16=case["kind"] != "f32")
        s["params"] = [p[0][:, 0].contiguous(), p[0][:, 1].contiguous(), *p[1:]]     # x, y, r, theta, v, c
        if op == "render":
            s["bg"] = torch.ones((H, W, 3), device="cuda")
        else:
            s.update(target=_target(case, seed), conf=_loop_conf(case), init=_Pool(case, seed))
    elif op == "fit":
        s["job"] = ImageFitter(*(q.cpu().numpy() for q in p), sets[0][5], Atlas(tmpl, case["kind"]),
                               _target(case, seed), torch.ones((H, W, 3), device="cuda"),
                               FitConfig(tile_size=case["tile"], alpha_max=case["alpha_max"]))
        s["host"] = torch.cat([q.reshape(-1) for q in p]).cpu().pin_memory()
        s["job"].capture()
    elif op == "psd":
        # the channel data of the file the program writes, and its directory: layer and four block sizes
        s.update(templates=tmpl, params=[p[0], p[1], p[2], torch.sigmoid(p[3]), torch.sigmoid(p[4])],
                 file=torch.zeros(case["N"] * 64 * max(H, W), dtype=torch.uint8).pin_memory())
    else:
        s["params"] = [q.requires_grad_() for q in p]
        s["up"] = _upstream(case, seed)
        if op == "dropin":
            s["tr"] = ctr.TileRasterizer(H, W, case["tile"], alpha_upper_bound=case["alpha_max"],
                                         num_primitives=case["N"], use_fp16=True)
            s["up"] = tuple(u.half() for u in s["up"])
            s.update(templates=tmpl, none=torch.empty(0, device="cuda"), lr=torch.ones(7, device="cuda"))
        else:
            s.update(atlas=Atlas(tmpl, case["kind"]), rz=Rasterizer(H, W, case["tile"], case["alpha_max"]))
            if case.get("c_blend"):
                maps = torch.rand(case["P"], case["th"], case["tw"], 3, device="cuda",
                                  generator=torch.Generator(device="cuda").manual_seed(seed + 3))
                s["maps"] = maps[s["sel"].long()]
    return s


# ---------------------------------------------------------------------------
# One pass
def run(s):
    op, case = s["op"], s["case"]
    if op == "render":
        with torch.no_grad():
            return s["renderer"].render_from_params(*s["params"], return_alpha=True, I_bg=s["bg"])
    if op == "loop":
        x, y, r, theta, v, c = (q.clone() for q in s["params"])
        out = s["renderer"].optimize_parameters(x, y, r, v, theta, c, s["target"], s["conf"], None, s["init"])
        return dict(zip("x y r v theta c".split(), out), loss=s["renderer"].last_loss)
    if op == "fit":
        job = s["job"]
        job.upload_params(s["host"])
        job.step()
        return dict(params=job.params_flat, m=job.adam_m, v=job.adam_v, loss=job.loss_dev)
    if op == "psd":
        m, r, th, v, c = s["params"]
        buf, bbox, sizes, offs = psd.export_layers(s["templates"], m, r, th, v, c, s["sel"], case["H"], case["W"],
                                                   alpha_max=case["alpha_max"])
        hs = sizes.cpu().numpy()
        keep = (hs[:, 0] > 1) & (hs[:, 1] > 1)
        blob, blocks, chosen = psd.encode_channel_blocks(buf, sizes, offs, hs, psd.ORDER_LAYER,
                                                         lambda a: np.nonzero(keep & (a > 0))[0][::-1])
        s["file"][:blob.numel()].copy_(blob)
        directory = np.full((case["N"], 5), -1, np.int64)
        directory[:len(chosen), 0], directory[:len(chosen), 1:] = chosen, blocks
        return s["file"], directory, bbox, sizes, offs
    if op == "dropin":
        out = s["tr"](*s["params"], s["none"], s["templates"], s["sel"], 0.0, s["lr"])
    elif op == "batch":
        out = rasterize_batch(*s["params"], s["sel"], s["atlas"], s["rz"])
    else:
        out = rasterize(*s["params"], s["sel"], s["atlas"], s["rz"], None, s.get("maps"), case.get("c_blend", 0.0))
    return [o.detach() for o in out], torch.autograd.grad(out, s["params"], s["up"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
def work(case):
    """Bytes: each input read once, each output written once.  Operations: 12 per (pixel, primitive) pair inside the
    primitive's square (texel coordinates and tests) and, per fragment that is still visible, 48 for the render and 96
    more for its gradients.  Pairs and fragments are the means of the parameter distributions: half extents
    log-uniform in [0.05, 0.3] of the canvas side, about half of a square covered, about 22 visible fragments at most
    above each other before a pixel is opaque; pairs behind an opaque pixel are not needed."""
    H, W, N, B, op = case["H"], case["W"], case["N"], case.get("B", 1), case["op"]
    side = float(min(H, W))
    r2 = (0.3 ** 2 - 0.05 ** 2) / (2 * math.log(6.0)) * side * side
    depth = N * 4 * r2 * 0.8 / (H * W)                 # squares over a pixel; a fifth lies outside the canvas
    seen = min(depth, 47.0)
    pairs, frags, px = H * W * seen, H * W * 0.47 * seen, H * W
    bytes_tex = case["P"] * case["th"] * case["tw"] * 4
    grad = op in ("grad", "dropin", "batch", "fit", "loop")
    flops = pairs * 12 * (2 if grad else 1) + frags * (144 if grad else 48)
    byts = bytes_tex + N * 36 + px * 16
    if op == "render":
        byts += px * 12
    elif op == "loop":
        n = case["iters"]
        flops, byts = n * flops, n * (bytes_tex + N * 36 + px * 24 + N * 8 * 4 * 5)
    elif op == "fit":
        byts = bytes_tex + N * 36 + px * 24 + N * 8 * 4 * 6
    elif op == "psd":
        crops = N * 4 * (0.25 * r2) * 2.25 * 0.85 * 4  # crops reach 1.5 r and are cut at the canvas
        flops, byts = crops / 4 * 30, bytes_tex + crops * 1.06
    else:
        byts += px * 16 + N * 32                        # image gradients in, parameter gradients out
        if case.get("c_blend"):
            byts += N * case["th"] * case["tw"] * 12
    return dict(bytes=float(byts * (B if op != "psd" else 1)), flops=float(flops * B))


# ---------------------------------------------------------------------------
# The same results in 64 bits: the compositing rule primitive by primitive on the pixels of its square
class _Exact:
    def __init__(self, H, W, templates, sel, alpha_max, maps=None, c_blend=0.0):
        self.H, self.W, self.sel, self.amax, self.maps, self.cb = H, W, sel, alpha_max, maps, c_blend
        self.Ht, self.Wt = templates.shape[1:]
        self.pad = torch.nn.functional.pad(templates.double(), (0, 1, 0, 1))    # neighbours outside read 0

    def _bind(self, m, r, th, v, c):
        """Per-primitive scalars from the parameter tensors."""
        m, r, th, v, c = (q.detach().double().cpu().numpy() for q in (m, r, th, v, c))
        self.p = (m, r, th)
        self.a0, self.col = self.amax / (1 + np.exp(-v)), 1 / (1 + np.exp(-c))
        self.sv, self.N = 1 / (1 + np.exp(-v)), len(r)

    def _entry(self, n, grad):
        """Mask of primitive n on its pixels and, with grad, its texel-space gradient and offsets; None off canvas."""
        (mx, my), r, th = self.p[0][n], self.p[1][n], self.p[2][n]
        s = r / (0.5 * max(self.Ht, self.Wt))
        hw, hh = 0.5 * self.Wt * s, 0.5 * self.Ht * s
        x0, x1 = max(0, math.ceil(mx - hw)), min(self.W - 1, math.floor(mx + hw))
        y0, y1 = max(0, math.ceil(my - hh)), min(self.H - 1, math.floor(my + hh))
        if x0 > x1 or y0 > y1:
            return None
        rinv = 1 / r if r > 1e-6 else 1e6
        hx, hy, ct, st = 0.5 * (self.Wt - 1), 0.5 * (self.Ht - 1), math.cos(th), math.sin(th)
        dx = torch.arange(x0, x1 + 1, device="cuda", dtype=torch.float64) - mx
        dy = (torch.arange(y0, y1 + 1, device="cuda", dtype=torch.float64) - my)[:, None]
        ex, ey = (ct * dx + st * dy) * (rinv * hx), (ct * dy - st * dx) * (rinv * hy)
        tx, ty = ex + hx, ey + hy
        ok = (tx >= 0) & (tx <= self.Wt - 1) & (ty >= 0) & (ty <= self.Ht - 1)
        fx, fy = tx.clamp(0, self.Wt - 1).floor(), ty.clamp(0, self.Ht - 1).floor()
        wx, wy = tx - fx, ty - fy
        row = self.Wt + 1
        i = (fy * row + fx).long()
        t = self.pad[self.sel[n]].reshape(-1)
        v00, v01, v10, v11 = t[i], t[i + 1], t[i + row], t[i + row + 1]
        top, bot = v00 + wx * (v01 - v00), v10 + wx * (v11 - v10)
        mask = (top + wy * (bot - top)).clamp(0, 1)
        mask = torch.where(ok & (mask > 1e-6), mask, 0.0)
        at = (slice(y0, y1 + 1), slice(x0, x1 + 1))
        col = self._colour(n, tx, ty)
        if not grad:
            return at, mask, col
        on = mask > 0
        gx = torch.where(on, (1 - wy) * (v01 - v00) + wy * (v11 - v10), 0.0)
        gy = torch.where(on, bot - top, 0.0)
        return at, mask, col, gx, gy, ex, ey, ct, st, rinv, hx, hy

    def _colour(self, n, tx, ty):
        col = [float(q) for q in self.col[n]]
        if self.maps is None:
            return col
        cm = self.maps[n].double().reshape(-1, 3)
        cx, cy = tx.clamp(0, self.Wt - 1), ty.clamp(0, self.Ht - 1)
        x0, y0 = cx.floor().long(), cy.floor().long()
        x1, y1 = (x0 + 1).clamp(max=self.Wt - 1), (y0 + 1).clamp(max=self.Ht - 1)
        fx, fy = (cx - x0)[..., None], (cy - y0)[..., None]
        at = lambda y, x: cm[y * self.Wt + x]
        c0 = at(y0, x0) * (1 - fx) + at(y0, x1) * fx
        c1 = at(y1, x0) * (1 - fx) + at(y1, x1) * fx
        q = c0 * (1 - fy) + c1 * fy
        return [(1 - self.cb) * col[k] + self.cb * q[..., k] for k in range(3)]

    def forward(self, *params):
        self._bind(*params)
        C = torch.zeros(3, self.H, self.W, device="cuda", dtype=torch.float64)
        T = torch.ones(self.H, self.W, device="cuda", dtype=torch.float64)
        for n in range(self.N):
            e = self._entry(n, False)
            if e is None:
                continue
            at, mask, col = e
            a = mask * float(self.a0[n])
            wt = T[at] * a
            for k in range(3):
                C[k][at] += wt * col[k]
            T[at] -= wt
        self.T = T
        return C.permute(1, 2, 0).contiguous(), 1 - T

    def backward(self, gC, gA):
        """The gradients (means, radii, rotations, opacity logits, colour logits) for the last forward()."""
        gC, gA, T = gC.double().permute(2, 0, 1).contiguous(), gA.double(), self.T.clone()
        Hs, Bt = torch.zeros_like(T), torch.ones_like(T)
        out = torch.zeros(self.N, 8, device="cuda", dtype=torch.float64)
        for n in reversed(range(self.N)):
            e = self._entry(n, True)
            if e is None:
                continue
            at, mask, col, gx, gy, ex, ey, ct, st, rinv, hx, hy = e
            a0 = float(self.a0[n])
            a = mask * a0
            om = 1 - a
            T[at] /= om
            Tk = T[at]
            g3 = gC[:, at[0], at[1]]
            gc = g3[0] * col[0] + g3[1] * col[1] + g3[2] * col[2]
            dl = Tk * (gc - Hs[at] + gA[at] * Bt[at])
            u, v, wt = dl * gx, dl * gy, a * Tk
            su, sv = u.sum(), v.sum()
            out[n, 0] = a0 * rinv * (st * hy * sv - ct * hx * su)
            out[n, 1] = -a0 * rinv * (st * hx * su + ct * hy * sv)
            out[n, 2] = -a0 * rinv * (u * ex + v * ey).sum()
            out[n, 3] = a0 * (u * ey * (hx / hy) - v * ex * (hy / hx)).sum()
            out[n, 4] = (1 - float(self.sv[n])) * (dl * a).sum()
            out[n, 5:8] = (g3 * wt).sum((1, 2))
            Hs[at] = om * Hs[at] + a * gc
            Bt[at] *= om
        s = torch.from_numpy(self.col).cuda()
        out[:, 5:8] *= s * (1 - s)
        return out[:, 0:2], out[:, 2], out[:, 3], out[:, 4], out[:, 5:8]

    def loss_and_grads(self, params, target, bg):
        C, A = self.forward(*params)
        d = C + (1 - A)[..., None] * bg - target.double()
        gC = d * (2.0 / d.numel())
        return (d * d).mean(), self.backward(gC, -(gC * bg).sum(-1))


def _adam(case, p, g, m, v, t, decay):
    """One torch.optim.Adam step in 64 bits; p, g, m, v: (N,8) x, y, r, theta, v, colours."""
    lr = torch.tensor([10, 10, 10, 1, 1.5 * 1000.0 / case["N"], 1, 1, 1], device="cuda", dtype=torch.float64)
    m.mul_(0.9).add_(0.1 * g)
    v.mul_(0.999).add_(0.001 * g * g)
    p -= 0.01 * decay * lr / (1 - 0.9 ** t) * m / (v.sqrt() / math.sqrt(1 - 0.999 ** t) + 1e-8)
    p[:, 0].clamp_(0, case["W"] - 1)
    p[:, 1].clamp_(0, case["H"] - 1)
    p[:, 2].clamp_(2, min(case["H"], case["W"]) // 4)


def _split(p):
    return p[:, 0:2], p[:, 2], p[:, 3], p[:, 4], p[:, 5:8]


def _blurred(t, sigma):
    if sigma <= 0:
        return t
    K = int(2 * round(3 * sigma) + 1)
    k = torch.exp(-0.5 * ((torch.arange(K, device="cuda", dtype=torch.float64) - K // 2) / sigma) ** 2)
    k = k / k.sum()
    return torch.nn.functional.conv2d(t.double()[:, None], (k[:, None] * k[None])[None, None], padding=K // 2)[:, 0]


def exact(case, seed):
    """run()'s floating outputs for prepare(case, seed)'s inputs, in 64 bits; None where it would take too long (a
    walk over tens of thousands of primitives) or where the outputs are bytes."""
    op, H, W, N = case["op"], case["H"], case["W"], case["N"]
    steps = case.get("iters", 1) * case.get("B", 1)
    if op == "psd" or N * steps > 9000 or N * steps * H * W > 9e9:
        return None
    _, t, sets = _inputs(case, seed)
    tmpl, sel = _dev(t), sets[0][5]
    if op == "render":
        C, A = _Exact(H, W, tmpl, sel, case["alpha_max"]).forward(*(_dev(q) for q in sets[0][:5]))
        return C + (1 - A)[..., None], A
    if op in ("fit", "loop"):
        p = torch.cat([_dev(q).double().reshape(N, -1) for q in sets[0][:5]], 1)
        m, v, target = torch.zeros_like(p), torch.zeros_like(p), _target(case, seed)
        if op == "fit":
            e = _Exact(H, W, tmpl, sel, case["alpha_max"])
            loss, g = e.loss_and_grads(_split(p), target, 1.0)
            _adam(case, p, torch.cat([q.reshape(N, -1) for q in g], 1), m, v, 1, 1.0)
            return dict(params=torch.cat([q.reshape(-1) for q in _split(p)]), m=m, v=v, loss=loss.view(1))
        n, pool, used = case["iters"], None, 0
        due = [it for it in range(n) if it and it % 3 == 0 and 1 < it < n - 1]
        q = _Pool(case, seed).reinitialize_subset(max(1, len(due) * N), None, "cuda")
        pool = torch.cat([q[0][:, None], q[1][:, None], q[2][:, None], q[4][:, None], q[3][:, None], q[5]], 1).double()
        for it in range(n):
            if it in due:
                low = (torch.sigmoid(p[:, 4].float()) < 0.3).nonzero()[:, 0]
                p[low] = pool[used:used + len(low)]
                used += len(low)
            e = _Exact(H, W, _blurred(tmpl, 2.0 * (1 - it / n)), sel, case["alpha_max"])
            loss, g = e.loss_and_grads(_split(p), target, 1.0)
            _adam(case, p, torch.cat([x.reshape(N, -1) for x in g], 1), m, v, it + 1, 0.99 ** it)
        return dict(x=p[:, 0], y=p[:, 1], r=p[:, 2], theta=p[:, 3], v=p[:, 4], c=p[:, 5:8], loss=float(loss))
    gC, gA = _upstream(case, seed)
    if op == "dropin":
        gC, gA = gC.half(), gA.half()
    maps = None
    if case.get("c_blend"):
        maps = torch.rand(case["P"], case["th"], case["tw"], 3, device="cuda",
                          generator=torch.Generator(device="cuda").manual_seed(seed + 3))[_dev(sel).long()]
    outs = []
    for b, q in enumerate(sets):
        e = _Exact(H, W, tmpl, sel, case["alpha_max"], maps, case.get("c_blend", 0.0))
        img = e.forward(*(_dev(a) for a in q[:5]))
        outs.append((img, e.backward(*((gC[b], gA[b]) if op == "batch" else (gC, gA)))))
    if op != "batch":
        return list(outs[0][0]), outs[0][1]
    return ([torch.stack([o[0][k] for o in outs]) for k in range(2)],
            tuple(torch.stack([o[1][k] for o in outs]) for k in range(5)))
