"""Performance cases: frames and gradient steps as a program that uses the
framework has it render them, through the package's public entry points.

Kinds of pass (`kind`):
  frame   one frame of a loaded scene (renderer.render_scene on the batched
          path), the framebuffer left on the device
  stream  one frame of an animation: new control points from host memory
          (Renderer.load_patches), the frame, the 8-bit display image in host
          memory (Renderer.read_image)
  grad    one optimization step's forward and backward through
          adjoint.render: image, control-point and amplitude gradients of a
          squared image loss

The per-pass path (path="plain") mirrors the reference's launch structure for
comparisons; programs render on the batched path, so the cases do.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from micropolis_gb300 import adjoint, scenes
from micropolis_gb300.renderer import Renderer, render_scene, renderer_for

DEFAULTS = dict(kind="frame", layout="heightfield", patches=64, width=1024, height=768, limit=8.0, dice=8,
                displaced=False, views=1, objects=1, criterion=0)


def _case(name: str = "", **kw) -> dict:
    c = dict(DEFAULTS, **kw)
    return dict(name=name, **c) if name else c


def listed() -> list:
    return [
        # an interactive preview of a small model: few patches, launch and latency count
        _case("preview_heightfield"),
        # an ordinary frame: thousands of patches of both types, uneven split depth
        _case("frame_mixed", layout="mixed", patches=4096, width=1920, height=1080),
        # the same with the finer dice grid (smoother shading)
        _case("frame_mixed_dice16", layout="mixed", patches=4096, width=1920, height=1080, dice=16),
        # a scene file's worth of objects, each a mesh of its own with its own transform, in an odd window
        _case("frame_objects", layout="objects", patches=1237, width=1000, height=760, objects=24),
        # Gregory patches with displacement (the export of subdivision models)
        _case("frame_gregory_displaced", layout="gregory", patches=1024, width=1280, height=720, displaced=True),
        # the reference's other bound criterion
        _case("frame_gpu_criterion", layout="mixed", patches=1024, width=1280, height=720, criterion=1),
        # a data set's worth of independent views in one launch
        _case("views64", layout="bezier", patches=10000, width=512, height=512, views=64),
        # the largest frame: fractal terrain at 4K with a fine split limit
        _case("terrain_4k", patches=512 * 512, width=3840, height=2160, limit=4.0, displaced=True),
        # an animation: upload, frame and display image through host memory
        _case("stream_mixed", kind="stream", layout="mixed", patches=2048, width=1920, height=1080),
        # fitting a small displaced surface to an image
        _case("grad_heightfield", kind="grad", patches=256, width=512, height=512, displaced=True),
        # fitting Gregory patches
        _case("grad_gregory", kind="grad", layout="gregory", patches=777, width=1280, height=720),
        # fitting terrain at 4K
        _case("grad_terrain_4k", kind="grad", patches=512 * 512, width=3840, height=2160, limit=4.0, displaced=True),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame", "frame", "frame", "stream", "grad", "grad"])
    # windows are whole 8-pixel tiles
    width = 8 * rng.randint(32, 240)
    height = 8 * rng.randint(24, 135)
    c = dict(kind=kind, width=width, height=height, displaced=rng.random() < 0.5,
             limit=rng.choice([8.0, 8.0, 10.0, 12.5]))
    layout = rng.choice(["heightfield", "mixed", "gregory", "bezier", "objects"])
    if kind == "grad":
        layout = rng.choice(["heightfield", "gregory", "bezier"])
    c["layout"] = layout
    if layout == "heightfield":
        c["patches"] = _log_int(rng, 3, 400) ** 2
        if rng.random() < 0.4:
            c.update(width=8 * rng.randint(160, 480), height=8 * rng.randint(90, 270), limit=rng.choice([4.0, 6.0]))
    else:
        c["patches"] = _log_int(rng, 60, 4096)
        if layout == "objects":
            c["objects"] = rng.randint(2, 100)
    if kind == "frame":
        c["criterion"] = 1 if rng.random() < 0.15 else 0
        if rng.random() < 0.3:
            c["dice"] = 16
        if layout == "bezier":
            # many views, each with its own scene and camera
            c.update(views=_log_int(rng, 2, 64), patches=_log_int(rng, 300, 6000), width=8 * rng.randint(16, 64),
                     height=8 * rng.randint(16, 64))
    return _case(**c)


# ---------------------------------------------------------------------------
# inputs


def _heightfield(rng, n: int) -> scenes.Mesh:
    """scenes.heightfield_mesh without its loop over patches; fractal heights for fine grids."""
    g = 3 * n + 1
    z = (rng.uniform(-0.2, 0.2, size=(g, g)) if n <= 32 else scenes.value_noise_fbm(rng, g))
    xs = np.linspace(-1.0, 1.0, g)
    grid = np.stack([*np.meshgrid(xs, xs, indexing="ij"), z], axis=-1).astype(np.float32)
    at = 3 * np.arange(n)[:, None] + np.arange(4)
    # patch a * n + b covers columns b and rows a of the control grid, point 4 i + j at (x = j, y = i)
    cp = grid[at[None, :, None, :], at[:, None, :, None]]
    return scenes.Mesh(scenes.BEZIER, np.ascontiguousarray(cp).reshape(n * n, 16, 3))


def _colour(rng) -> tuple:
    return (*(float(x) for x in rng.uniform(0.2, 0.95, 3)), 1.0)


def _scene(case: dict, seed: int) -> scenes.Scene:
    rng = np.random.default_rng(seed)
    n, layout = case["patches"], case["layout"]
    if layout == "heightfield":
        side = max(1, math.isqrt(n))
        eye = np.array((0.0, -2.5, 1.5) if case["limit"] > 4.0 else (0.0, -1.9, 0.9)) + rng.uniform(-0.05, 0.05, 3)
        draws = [scenes.Draw(_heightfield(rng, side), scenes.look_at(eye, (0, 0, 0), (0, 0, 1)), _colour(rng))]
    elif case["views"] > 1:
        draws = []
        counts = np.exp(rng.uniform(np.log(max(1, n // 100)), np.log(n), size=case["views"])).astype(int)
        for v, eye in enumerate(scenes.fibonacci_sphere(case["views"], 15.0)):
            up = (0, 0, 1) if abs(eye[2]) < 14.5 else (0, 1, 0)
            draws.append(scenes.Draw(scenes.scattered_patches(rng, int(counts[v]), gregory=False),
                                     scenes.look_at(eye, (0, 0, 0), up), _colour(rng), view=v))
    else:
        eye = np.array([0.6, -0.8, 0.35]) + rng.uniform(-0.05, 0.05, 3)
        mv = scenes.look_at(eye / np.linalg.norm(eye) * scenes.MIXED_CAMERA_DISTANCE, (0, 0, 0), (0, 0, 1))
        if layout == "mixed":
            parts = [(n // 2, False), (n - n // 2, True)]
        elif layout == "objects":
            k = case["objects"]
            parts = [(n * (i + 1) // k - n * i // k, i % 2 == 1) for i in range(k)]
        else:
            parts = [(n, layout == "gregory")]
        draws = []
        for count, gregory in parts:
            m = mv
            if layout == "objects":
                move = np.eye(4, dtype=np.float32)
                move[:3, 3] = rng.uniform(-2, 2, 3)
                m = (mv.reshape(4, 4).T @ move).T.reshape(16).astype(np.float32)
            draws.append(scenes.Draw(scenes.scattered_patches(rng, max(1, count), gregory), m, _colour(rng)))
    opts = dict(bound_n_split_limit=case["limit"], reyes_patch_size=case["dice"], batch_views=case["views"],
                displacement=int(case["displaced"]), bound_criterion=case["criterion"])
    return scenes.Scene(case["layout"], case["width"], case["height"], draws, options=opts, seed=seed)


class _DeviceArray:
    """A device buffer of the renderer, for torch.as_tensor (the tensor keeps
    this object, and with it the renderer that owns the buffer, alive)."""

    def __init__(self, owner: Renderer, ptr: int, shape: tuple, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _framebuffer(r: Renderer):
    colour, depth = r.framebuffer_ptrs()
    n = r.width * r.height * r.views
    return (torch.as_tensor(_DeviceArray(r, colour, (n, 4), "<f4"), device="cuda"),
            torch.as_tensor(_DeviceArray(r, depth, (n,), "<i4"), device="cuda"))


def _target(case: dict, seed: int) -> torch.Tensor:
    """The image to fit, in framebuffer order: smooth variation in the range of the shaded colours."""
    g = torch.Generator().manual_seed(seed)
    coarse = torch.rand((1, 3, 9, 16), generator=g).cuda() * 0.6 + 0.1
    h, w = case["height"], case["width"]
    img = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=True)[0]
    return img.reshape(3, h // 8, 8, w // 8, 8).permute(1, 3, 2, 4, 0).reshape(h * w, 3).contiguous()


AMPLITUDE = 1.1


def prepare(case: dict, seed: int) -> dict:
    sc = _scene(case, seed)
    if case["kind"] == "grad":
        dr = adjoint.DiffRenderer(sc)
        cp = torch.tensor(sc.draws[0].mesh.cp, device="cuda", requires_grad=True)
        amp = torch.tensor(AMPLITUDE, device="cuda", requires_grad=True)
        return dict(kind="grad", dr=dr, cp=cp, amp=amp, target=_target(case, seed))
    r = renderer_for(sc, "batched")
    handles = list(range(1, len(sc.draws) + 1))
    s = dict(kind=case["kind"], r=r, scene=sc, handles=handles, fb=_framebuffer(r))
    for h, d in zip(handles, sc.draws):
        r.load_patches(h, d.mesh.cp, d.mesh.type)
    return s


def run(state: dict):
    if state["kind"] == "grad":
        cp, amp = state["cp"], state["amp"]
        img = adjoint.render(cp, amp, state["dr"])
        loss = ((img[:, :3] - state["target"]) ** 2).sum()
        g_cp, g_amp = torch.autograd.grad(loss, (cp, amp))
        return img.detach(), g_cp, g_amp
    r, sc = state["r"], state["scene"]
    if state["kind"] == "stream":
        for h, d in zip(state["handles"], sc.draws):
            r.load_patches(h, d.mesh.cp, d.mesh.type)
    render_scene(r, sc, state["handles"])
    if state["kind"] == "stream":
        return r.read_image()
    return state["fb"]


def _points(case: dict) -> int:
    """Control points of all patches (the views' counts are log-uniform over two decades)."""
    n = case["patches"]
    if case["layout"] == "heightfield":
        return 16 * max(1, math.isqrt(n)) ** 2
    if case["views"] > 1:
        return int(16 * case["views"] * n * 0.99 / math.log(100))
    return {"bezier": 16, "gregory": 20}.get(case["layout"], 18) * n


def work(case: dict) -> dict:
    px = case["width"] * case["height"] * case["views"]
    pts = _points(case)
    # A sub-patch covers at most limit x limit pixels, so the frame has at
    # least (surface layers a pixel sees, both facings) * pixels / limit^2 of
    # them, each (dice + 1)^2 vertices of about 230 operations (the patch
    # sum, modelview and projection), and 12 sines more when displaced.
    layers = 0.4 if case["layout"] == "heightfield" else 5.0 * pts / 18 / 4096 / case["views"]
    subs = max(pts / 18, layers * px / case["limit"] ** 2)
    flops = subs * (case["dice"] + 1) ** 2 * (230 + (12 * 20 if case["displaced"] else 0))
    if case["kind"] == "stream":
        return dict(bytes=12 * pts + 3 * px, flops=flops)
    if case["kind"] == "grad":
        # control points in, image out; image gradient in, control-point gradients out;
        # four vertices recomputed and differentiated per covered pixel
        return dict(bytes=2 * (12 * pts + 16 * px), flops=flops + 0.3 * px * 4 * (400 + (900 if case["displaced"] else 0)))
    return dict(bytes=12 * pts + 20 * px, flops=flops)


# ---------------------------------------------------------------------------
# The same pass in plain torch: the reference's bound-and-split decisions in
# IEEE single precision (they choose the sub-patches), everything after them
# in 64 bits.


def _spline32(t, p):
    """Cubic Bernstein sum in single precision, left to right; t (m,), p four (m, 3)."""
    s = 1.0 - t
    w = (s * s * s, 3.0 * s * s * t, 3.0 * s * t * t, t * t * t)
    out = w[0][:, None] * p[0]
    for k in (1, 2, 3):
        out = out + w[k][:, None] * p[k]
    return out


def _point32(P, gregory: bool, su, sv):
    if not gregory:
        return _spline32(sv, [_spline32(su, [P[:, 4 * i + j] for j in range(4)]) for i in range(4)])
    u, v = sv, su
    a, b = 1.0 - u, 1.0 - v

    def blend(x, A, y, B, den):
        return (x[:, None] * P[:, A] + y[:, None] * P[:, B]) / den[:, None]
    F0, F1 = blend(u, 12, v, 16, u + v), blend(a, 17, v, 13, a + v)
    F2, F3 = blend(a, 18, b, 14, 2.0 - u - v), blend(u, 19, b, 15, 1.0 + u - v)
    rows = [(P[:, 0], P[:, 8], P[:, 7], P[:, 3]), (P[:, 4], F0, F3, P[:, 11]), (P[:, 9], F1, F2, P[:, 6]),
            (P[:, 1], P[:, 5], P[:, 10], P[:, 2])]
    return _spline32(v, [_spline32(u, r) for r in rows])


def _skip_nan(fn, a, b):
    """minimum / maximum that keep b where a is NaN (the bound's comparisons)."""
    return torch.where(torch.isnan(a), b, fn(a, b))


def _subpatches(cp, gregory: bool, mv, sc):
    """The emitted (patch, range) list of one draw."""
    W, H, near, limit = sc.width, sc.height, np.float32(sc.near), sc.options["bound_n_split_limit"]
    fy = np.float32(1) / np.float32(math.tan(sc.fovy * math.pi / 360))
    fx = fy / np.float32(W / H)
    vx, vy = np.float32(W / 2), np.float32(H / 2)
    kx, ky, vx, vy, near = float(fx * vx), float(fy * vy), float(vx), float(vy), float(near)
    pid = torch.arange(len(cp), device="cuda")
    r = torch.tensor([0.0, 0.0, 1.0, 1.0], device="cuda").repeat(len(cp), 1)
    m = torch.tensor(mv, device="cuda")
    out = []
    for depth in range(25):
        if not len(pid):
            break
        P = cp[pid]
        ps = [[None] * 3 for _ in range(3)]
        for iu in range(3):
            for iv in range(3):
                q = _point32(P, gregory, r[:, 1] + (r[:, 3] - r[:, 1]) * iv * 0.5,
                             r[:, 0] + (r[:, 2] - r[:, 0]) * iu * 0.5)
                x, y, z = q[:, :1], q[:, 1:2], q[:, 2:]
                ps[iu][iv] = (m[0:3] * x + m[4:7] * y) + (m[8:11] * z + m[12:15])
        del P
        inf = torch.full_like(r[:, :3], math.inf)
        lo, hi = inf, -inf
        for q in (q for c in ps for q in c):
            lo, hi = _skip_nan(torch.minimum, q, lo), _skip_nan(torch.maximum, q, hi)

        def dist(a, b):
            d = (b - a) * (b - a)
            return torch.sqrt((d[:, 0] + d[:, 1]) + d[:, 2])
        vlen = hlen = torch.zeros_like(r[:, 0])
        for i in range(3):
            vlen = _skip_nan(torch.maximum, dist(ps[0][i], ps[1][i]) + dist(ps[1][i], ps[2][i]), vlen)
            hlen = _skip_nan(torch.maximum, dist(ps[i][0], ps[i][1]) + dist(ps[i][1], ps[i][2]), hlen)
        n, f = torch.clamp(-hi[:, 2], min=near), -lo[:, 2]

        def screen(v, k, c, use_n):
            return (v / torch.where(use_n, n, f)) * k + c
        x0, x1 = screen(lo[:, 0], kx, vx, lo[:, 0] < 0), screen(hi[:, 0], kx, vx, hi[:, 0] > 0)
        y0, y1 = screen(lo[:, 1], ky, vy, lo[:, 1] < 0), screen(hi[:, 1], ky, vy, hi[:, 1] > 0)
        cull = (f < near) | (x0 > W - 1 + 32.0) | (x1 < -32.0) | (y0 > H - 1 + 32.0) | (y1 < -32.0)
        emit = ~cull & (lo[:, 2] < 0) & (x1 - x0 < limit) & (y1 - y0 < limit)
        out.append((pid[emit], r[emit]))
        split = ~cull & ~emit & (depth <= 23)
        by_y = (vlen < hlen)[split]
        pid, r = pid[split], r[split]
        cx, cy = (r[:, 0] + r[:, 2]) * 0.5, (r[:, 1] + r[:, 3]) * 0.5
        low, high = r.clone(), r.clone()
        low[:, 2], high[:, 0] = torch.where(by_y, r[:, 2], cx), torch.where(by_y, r[:, 0], cx)
        low[:, 3], high[:, 1] = torch.where(by_y, cy, r[:, 3]), torch.where(by_y, cy, r[:, 1])
        pid, r = torch.cat([pid, pid]), torch.cat([low, high])
    return torch.cat([p for p, _ in out]), torch.cat([q for _, q in out])


def _weights(gregory: bool, tx, ty):
    """Weight of every control point at (tx, ty): (..., 16 | 20), 64 bits."""
    def bern(t):
        s = 1.0 - t
        return (s * s * s, 3.0 * s * s * t, 3.0 * s * t * t, t * t * t)
    b, c = bern(tx), bern(ty)
    w = [x * y for x in b for y in c]
    if not gregory:
        return torch.stack(w, -1)
    u, v = tx, ty
    faces = {5: (u, 12, v, 16, u + v), 6: (1 - u, 17, v, 13, 1 - u + v), 10: (1 - u, 14, 1 - v, 18, 2 - u - v),
             9: (u, 19, 1 - v, 15, 1 + u - v)}
    slot = [0, 4, 9, 1, 8, -1, -1, 5, 7, -1, -1, 10, 3, 11, 6, 2]
    full = [None] * 20
    for k in range(16):
        if k not in faces:
            full[slot[k]] = w[k]
            continue
        x, A, y, B, den = faces[k]
        safe = torch.where(den == 0, torch.ones_like(den), den)
        full[A] = torch.where(den == 0, torch.zeros_like(den), w[k] * x / safe)
        full[B] = torch.where(den == 0, torch.zeros_like(den), w[k] * y / safe)
    return torch.stack(full, -1)


def _eye(points, mv, amp):
    """Modelview and (amp is not None) displacement of (..., 3) points."""
    m = torch.tensor(mv, device="cuda", dtype=torch.float64).reshape(4, 4)
    p = points @ m[:3, :3] + m[3, :3]
    if amp is None:
        return p
    x, y, z = p.unbind(-1)
    for k, a in ((10.0, 0.04), (14.0, 0.02), (22.0, 0.01)):
        a = a * amp
        x = x + torch.sin(k * y) * a
        y = y + torch.sin(k * x) * a
        z = z + torch.sin(k * y) * torch.sin(6.0 * x) * a
    return torch.stack([x, y, z], -1)


def _diffuse(p):
    """Diffuse factor of quads from four eye positions, a (..., 4, 3) tensor."""
    du = 0.5 * (p[..., 1, :] - p[..., 0, :] + p[..., 3, :] - p[..., 2, :])
    dv = 0.5 * (p[..., 2, :] - p[..., 0, :] + p[..., 3, :] - p[..., 1, :])
    n = torch.linalg.cross(dv, du)
    light = torch.tensor([4.0, 3.0, 8.0], device="cuda", dtype=torch.float64) / math.sqrt(89.0)
    length = n.norm(dim=-1).clamp(min=1e-300)
    return ((n @ light) / length).clamp(min=0.0)


def _raster(keys, pos, sc, base: int, view: int):
    """Depth|id minimum of the quads of sub-patches `base`... whose dice vertices are pos (m, G, G, 3) [v, u]."""
    W, H = sc.width, sc.height
    th = np.tan(np.float32(sc.fovy * math.pi / 180) / np.float32(2))
    mx, my = float(np.float32(1) / (np.float32(W / H) * th)), float(np.float32(1) / th)
    zn, zf = np.float32(sc.near), np.float32(10000.0)
    mz, mw = float(-(zf + zn) / (zf - zn)), float(-(np.float32(2) * zf * zn) / (zf - zn))
    x, y, z = pos.unbind(-1)
    ix = (x * mx / -z * (W * 32.0) + W * 32).trunc().clamp(-2**31, 2**31 - 1).to(torch.int64)
    iy = (y * my / -z * (H * 32.0) + H * 32).trunc().clamp(-2**31, 2**31 - 1).to(torch.int64)
    dep = (mz * z + mw) / -z
    n, ps = len(pos), pos.shape[1] - 1

    def corners(a):
        return torch.stack([a[:, :-1, :-1], a[:, :-1, 1:], a[:, 1:, :-1], a[:, 1:, 1:]], -1).reshape(n * ps * ps, 4)
    X, Y = corners(ix), corners(iy)
    e = (X - X[:, :1], Y - Y[:, :1])
    wind = (e[0][:, 1] * e[1][:, 3] - e[0][:, 3] * e[1][:, 1] < 0) | \
        (e[0][:, 3] * e[1][:, 2] - e[0][:, 2] * e[1][:, 3] < 0)
    x0, x1 = ((X.amin(1) + 63) >> 6).clamp(min=0), (X.amax(1) >> 6).clamp(max=W - 1)
    y0, y1 = ((Y.amin(1) + 63) >> 6).clamp(min=0), (Y.amax(1) >> 6).clamp(max=H - 1)
    live = torch.nonzero(wind & (x0 <= x1) & (y0 <= y1))[:, 0]
    X, Y, D = X[live], Y[live], corners(dep)[live]
    x0, x1, y0, y1 = x0[live], x1[live], y0[live], y1[live]
    ids = live + base * ps * ps
    gx = W // 8
    for oy in range(int((y1 - y0).max()) + 1 if len(live) else 0):
        rows = torch.nonzero(y0 + oy <= y1)[:, 0]
        for ox in range(int((x1 - x0)[rows].max()) + 1):
            k = rows[x0[rows] + ox <= x1[rows]]
            px, py = x0[k] + ox, y0[k] + oy
            best = torch.full((len(k),), 2.0, device="cuda", dtype=torch.float64)
            for tri in ((0, 1, 3), (0, 3, 2)):
                A, B, d = X[k][:, tri], Y[k][:, tri], D[k][:, tri]
                An, Bn = A.roll(-1, 1), B.roll(-1, 1)
                dx, dy = Bn - B, A - An
                V = dx * (px[:, None] * 64 - A) + dy * (py[:, None] * 64 - B)
                C = -((dx > 0) | ((dx == 0) & (dy > 0))).to(torch.int64)
                ok = (V > C).all(1)
                area = (dx[:, 1] * (A[:, 0] - A[:, 1]) + dy[:, 1] * (B[:, 0] - B[:, 1])).to(torch.float64)
                t = (V.roll(-1, 1) * d).sum(1) / torch.where(area == 0, torch.ones_like(area), area)
                best = torch.where(ok, torch.minimum(best, t.clamp(max=1.0)), best)
            hit = best <= 1.0
            k, px, py = k[hit], px[hit], py[hit]
            idepth = ((best[hit] * 0.005).clamp(0.0, 1.0) * 2.0**31).to(torch.int64)
            at = (px // 8 + gx * (py // 8)) * 64 + px % 8 + (py % 8) * 8 + view * W * H
            keys.scatter_reduce_(0, at, (idepth << 32) | ids[k], "amin")


def exact(case: dict, seed: int):
    if case["kind"] == "stream":
        return None      # bytes of the display image: whole numbers
    if case["criterion"]:
        return None      # its decisions are taken in fused single precision: no 64-bit value
    sc = _scene(case, seed)
    ps = case["dice"]
    amp = AMPLITUDE if case["kind"] == "grad" else 1.0
    shift = amp if case["displaced"] else None
    keys = torch.full((sc.width * sc.height * case["views"],), 0x7fffffffffffffff, device="cuda", dtype=torch.int64)
    lists, base = [], 0
    t = torch.arange(ps + 1, device="cuda", dtype=torch.float64) / ps
    for d in sc.draws:
        cp = torch.tensor(d.mesh.cp, device="cuda")
        gregory = d.mesh.type == scenes.GREGORY
        pid, rg = _subpatches(cp, gregory, d.mv, sc)
        lists.append((base, pid, rg))
        step = (1 << 21) // (ps + 1) ** 2
        for i in range(0, len(pid), step):
            p, r = pid[i:i + step], rg[i:i + step].double()
            tx = (r[:, 0:1] + (r[:, 2:3] - r[:, 0:1]) * t)[:, None, :].expand(-1, ps + 1, -1)
            ty = (r[:, 1:2] + (r[:, 3:4] - r[:, 1:2]) * t)[:, :, None].expand(-1, -1, ps + 1)
            w = _weights(gregory, tx, ty).reshape(len(p), (ps + 1) ** 2, -1)
            pos = _eye(torch.bmm(w, cp[p].double()), d.mv, shift).reshape(len(p), ps + 1, ps + 1, 3)
            _raster(keys, pos, sc, base + i, d.view)
        base += len(pid)
    # the winning quads' colours from their four vertices
    covered = torch.nonzero(keys != 0x7fffffffffffffff)[:, 0]
    win = keys[covered] & 0xffffffff
    img = torch.empty((len(keys), 4), device="cuda", dtype=torch.float64)
    img[:] = torch.tensor([*(c ** 2.2 for c in (0.1, 0.1, 0.7)), 1000.0], device="cuda", dtype=torch.float64)
    grad = case["kind"] == "grad"
    corner = torch.tensor([[0, 0], [1, 0], [0, 1], [1, 1]], device="cuda", dtype=torch.float64)
    for d, (first, pid, rg) in zip(sc.draws, lists):
        mine = (win >= first * ps * ps) & (win < (first + len(pid)) * ps * ps)
        at, q = covered[mine], win[mine] - first * ps * ps
        s, q = q // (ps * ps), q % (ps * ps)
        cp = torch.tensor(d.mesh.cp, device="cuda", dtype=torch.float64, requires_grad=grad)
        a = torch.tensor(amp, device="cuda", dtype=torch.float64, requires_grad=grad)
        r = rg[s].double()
        tx = r[:, 0:1] + (r[:, 2:3] - r[:, 0:1]) * ((q % ps)[:, None] + corner[:, 0]) / ps
        ty = r[:, 1:2] + (r[:, 3:4] - r[:, 1:2]) * ((q // ps)[:, None] + corner[:, 1]) / ps
        w = _weights(d.mesh.type == scenes.GREGORY, tx, ty)
        m = _diffuse(_eye(torch.bmm(w, cp[pid[s]]), d.mv, a if case["displaced"] else None))
        dc = torch.tensor(d.color, device="cuda", dtype=torch.float64)
        ambient = torch.tensor([0.015, 0.015, 0.015, 1.0], device="cuda", dtype=torch.float64)
        colour = m[:, None] * dc + ambient * dc
        img[at] = colour.detach()
        if grad:
            loss = ((colour[:, :3] - _target(case, seed).double()[at]) ** 2).sum()
            g_cp, g_amp = torch.autograd.grad(loss, (cp, a), allow_unused=True)
            return img, g_cp, torch.zeros_like(a) if g_amp is None else g_amp
    return img, None
