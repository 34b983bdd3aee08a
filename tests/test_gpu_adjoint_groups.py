"""The adjoint's sums over a warp's patches: one patch for all pixels, a few,
and as many as pixels; both patch types and dice grids, with and without
displacement; control points never seen and frames nobody covers.  Gradients
against the oracle's analytic FP64 ones at the repository's bar of 1e-3 (the
micropolygons' edges are at least 4e-3 of the positions' size, as on the
16x16 heightfield that bar was set on)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 128, 96
GRAD_RTOL = 1e-3


def _grid(nx, ny, gregory=False, seed=0, depth=-1.0):
    """nx x ny patches, each with its own bumps, tiling a wall that covers most of the frame."""
    from micropolis_gb300 import scenes
    rng = np.random.default_rng(seed)
    half = np.tan(np.radians(30.0)) * 0.9
    t = np.arange(4) / 3.0
    cp = []
    for a in range(nx):
        for b in range(ny):
            x = (-1 + 2 * (a + t) / nx) * half * W / H
            y = (-1 + 2 * (b + t) / ny) * half
            X, Y = np.meshgrid(x, y)
            cp.append(np.stack([X, Y, depth + rng.normal(size=(4, 4)) * 0.15 / max(nx, ny)], -1).reshape(16, 3))
    cp = np.array(cp, np.float32)
    m = scenes.Mesh(scenes.GREGORY, np.ascontiguousarray(cp[:, scenes.BEZIER_TO_GREGORY])) if gregory else \
        scenes.Mesh(scenes.BEZIER, cp)
    return scenes.Scene("grid", W, H, [scenes.Draw(m, np.eye(4, dtype=np.float32).reshape(16), (0.9, 0.6, 0.4, 1.0))])


CASES = {
    "one_patch": ((1, 1), {}),
    "one_gregory": ((1, 1, True), {}),
    "few": ((5, 4), {}),
    "few_gregory": ((5, 4, True), {}),
    "few_gregory_displaced": ((5, 4, True), dict(displacement=1)),
    "few_displaced": ((5, 4), dict(displacement=1)),
    "few_dice16": ((5, 4), dict(reyes_patch_size=16, bound_n_split_limit=16.0)),
    "patch_per_pixel": ((61, 47), {}),
    "patch_per_pixel_gregory": ((61, 47, True), {}),
    "behind": ((2, 2, False, 0, 3.0), {}),
}


@pytest.mark.parametrize("name", list(CASES))
def test_gradients_match_fp64(built, cuda, name):
    torch = cuda
    from micropolis_gb300 import adjoint
    from oracle import oracle
    args, over = CASES[name]
    sc = _grid(*args)
    sc.options.update(over)
    dr = adjoint.DiffRenderer(sc)
    cp = torch.tensor(sc.draws[0].mesh.cp, device="cuda", requires_grad=True)
    amp = torch.tensor(0.8, device="cuda", requires_grad=True)
    target = torch.tensor(np.random.default_rng(3).uniform(0, 1, (W * H, 4)).astype(np.float32), device="cuda")
    img = adjoint.render(cp, amp, dr)
    ((img - target) ** 2).sum().backward()
    torch.cuda.synchronize()
    win = dr.r.visibility(0)
    _, pid, rng = dr.r.subpatches()
    _, g_ref, ga_ref = oracle.loss_fp64(sc, pid, rng, win, target.cpu().numpy(), cp.detach().double().cpu().numpy(), 0.8)
    g = cp.grad.double().cpu().numpy()
    assert np.linalg.norm(g - g_ref) <= GRAD_RTOL * np.linalg.norm(g_ref)
    assert abs(float(amp.grad) - ga_ref) <= GRAD_RTOL * max(abs(ga_ref), 1e-3 * np.linalg.norm(g_ref))
    if name == "behind":
        assert not g.any()
    # patches without a pixel get exactly nothing
    seen = np.unique(pid[win[win >= 0] // sc.options.get("reyes_patch_size", 8) ** 2])
    unseen = np.setdiff1d(np.arange(len(g)), seen)
    assert not g[unseen].any()
    dr.r.close()
