"""The fused kernel's shortcuts where they could go wrong, against the oracle
at every pixel: quads that end exactly at the frame's left edge (the one place
where a small quad asks for its 8x8 block bound), strips of quads that leave
the frame on each side, quads too large for the fast raster (their tiles come
from the block bound), backface culling off, groups with more runs of equal
draws than stage their matrices, partial groups, and face control points that
are not finite (NaN face points are zeroed)."""
import numpy as np
import pytest

from helpers import assert_identical_to_oracle

pytestmark = pytest.mark.gpu

W, H, NEAR_Z = 192, 128, 1.0
EDGE = np.tan(np.radians(30.0))                 # half height of the view at z = -1
PX = 2 * EDGE / H                               # a pixel at z = -1


def _scene(meshes, colors=None, **opts):
    from micropolis_gb300 import scenes
    eye = np.eye(4, dtype=np.float32).reshape(16)
    draws = [scenes.Draw(m, eye, (0.3 + 0.05 * (k % 10), 0.8, 0.5, 1.0)) for k, m in enumerate(meshes)]
    return scenes.Scene("edges", W, H, draws, options=opts)


def _wall(x0, x1, y0, y1, seed=0, bump=0.002, gregory=False):
    """A patch facing the eye over pixels [x0, x1] x [y0, y1] (framebuffer coordinates)."""
    from micropolis_gb300 import scenes
    t = np.arange(4) / 3.0
    X, Y = np.meshgrid((x0 + (x1 - x0) * t - W / 2) * PX, (y0 + (y1 - y0) * t - H / 2) * PX)
    z = -NEAR_Z + bump * np.random.default_rng(seed).normal(size=(4, 4))
    cp = np.stack([X * -z, Y * -z, z], -1).reshape(1, 16, 3).astype(np.float32)
    if gregory:
        return scenes.Mesh(scenes.GREGORY, cp[:, scenes.BEZIER_TO_GREGORY])
    return scenes.Mesh(scenes.BEZIER, cp)


def _left_edge():
    # right ends within a sixty-fourth of a pixel of x = 0, on both sides of it
    return [_wall(-20, d / 64.0, 8 * k, 8 * k + 7, seed=k, bump=0.0)
            for k, d in enumerate((-2, -1.01, -0.99, -0.5, 0, 0.5, 0.99, 1.01, 2, 63, 64, 65))]


def _around():
    return [_wall(-15, 20, -10, 40, 1), _wall(W - 20, W + 17, 10, 60, 2), _wall(30, 90, H - 12, H + 21, 3),
            _wall(60, 120, -25, 12, 4, gregory=True), _wall(-5, W + 5, 50, 70, 5)]


def _nonfinite():
    out = []
    for k, v in enumerate((np.nan, np.inf, -np.inf, 3e38)):
        m = _wall(10 + 40 * k, 45 + 40 * k, 20, 60, k, gregory=True)
        m.cp[0, 12 + 2 * k, 1] = v
        out.append(m)
    return out + [_wall(10, 100, 70, 120, 9, gregory=True)]


CASES = {
    "left_edge": (_left_edge, {}),
    "around": (_around, {}),
    "around_no_backface": (_around, dict(backface_culling=0)),
    "large_quads": (_around, dict(bound_n_split_limit=400.0)),
    "large_quads_no_backface": (_around, dict(bound_n_split_limit=400.0, backface_culling=0)),
    "many_draws": (lambda: [_wall(5 * k, 5 * k + 9, 3 * k, 3 * k + 11, k, gregory=k % 3 == 1) for k in range(37)], {}),
    "one_subpatch": (lambda: [_wall(10, 14, 10, 14)], {}),
    "displaced": (_around, dict(displacement=1, displacement_amplitude=0.4)),
    "nonfinite_faces": (_nonfinite, dict(max_split_depth=7)),
}


@pytest.mark.parametrize("dice", [8, 16])
@pytest.mark.parametrize("name", list(CASES))
def test_frame_identical_to_oracle(built, cuda, name, dice):
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    make, over = CASES[name]
    sc = _scene(make(), reyes_patch_size=dice, **over)
    r = renderer_for(sc, "batched")
    render_scene(r, sc)
    assert_identical_to_oracle(r, sc, oracle.make_params(sc))
    r.close()
