"""The dice's plain run and its general one, against the oracle at every
pixel: Gregory patches whose face points are not finite (one, and all, of the
eight), with and without displacement, corner vertices where a face blend is
0 / 0, and corners so deep in their patch that 1 + u rounds to 1 and the
blend's denominator is 0 while its numerator is not; vertices on the eye
plane; positions too large for the packed displacement."""
import numpy as np
import pytest

from helpers import assert_identical_to_oracle
from test_gpu_raster_edges import _scene, _wall

pytestmark = pytest.mark.gpu


def _faces(values, which):
    out = []
    for k, v in enumerate(values):
        m = _wall(8 + 44 * k, 44 + 44 * k, 15, 60, k, gregory=True)
        m.cp[0, which(k), :] = v
        out.append(m)
    return out + [_wall(20, 150, 70, 120, 9, gregory=True)]


def _corners(turn, long):
    """A Gregory patch with one corner in the middle of the frame and one side `long` units away."""
    from micropolis_gb300 import scenes
    t = np.arange(4) / 3.0
    X, Y = np.meshgrid(t, t)
    uv = [(X, Y), (1 - Y, X), (1 - X, 1 - Y), (Y, 1 - X)][turn % 4]
    x, y = (uv[0] * long, uv[1] * 0.4) if turn < 4 else (uv[0] * 0.4, uv[1] * long)
    cp = np.stack([x, y, -1.0 + 0.01 * np.sin(np.arange(16.0)).reshape(4, 4) * (long < 10)], -1)
    if turn % 4 in (1, 2):
        cp[..., 0] -= cp[..., 0].max()
    if turn % 4 in (2, 3):
        cp[..., 1] -= cp[..., 1].max()
    return scenes.Mesh(scenes.GREGORY, cp.reshape(1, 16, 3)[:, scenes.BEZIER_TO_GREGORY].astype(np.float32))


def _eye_plane():
    """Patches through the eye plane whose vertices lie exactly on it."""
    from micropolis_gb300 import scenes
    t = np.arange(4) / 3.0
    out = []
    for k, gregory in enumerate((False, True)):
        X, Y = np.meshgrid(t - 0.5, 0.3 * t + 0.1 * k)
        cp = np.stack([X, Y - 0.2, X * 2 - 0.25 * k], -1).reshape(1, 16, 3).astype(np.float32)
        out.append(scenes.Mesh(scenes.GREGORY, cp[:, scenes.BEZIER_TO_GREGORY]) if gregory else scenes.Mesh(scenes.BEZIER, cp))
    return out


def _far():
    m = _wall(20, 100, 20, 90, 3)
    g = _wall(60, 150, 30, 110, 4, gregory=True)
    for k in (m, g):
        k.cp *= np.float32(1e6)
    return [m, g]


ODD = (np.nan, np.inf, -np.inf, 3e38)
GPU = dict(bound_criterion=1, max_split_depth=8)   # its bound zeroes NaN faces too, so the sub-patches reach the dice
CASES = {
    "one_face": (lambda: _faces(ODD, lambda k: 12 + 2 * k), GPU),
    "all_faces": (lambda: _faces(ODD, lambda k: slice(12, 20)), GPU),
    "corners": (lambda: [_corners(k, 0.5) for k in range(8)], {}),
    "deep_corners": (lambda: [_corners(k, 6e5) for k in range(8)], dict(max_split_depth=30)),
    "eye_plane": (_eye_plane, dict(max_split_depth=12)),
    "far": (_far, {}),
}


@pytest.mark.parametrize("dice", [8, 16])
@pytest.mark.parametrize("displacement", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_frame_identical_to_oracle(built, cuda, name, displacement, dice):
    from micropolis_gb300.renderer import render_scene, renderer_for
    make, over = CASES[name]
    sc = _scene(make(), reyes_patch_size=dice, displacement=displacement, displacement_amplitude=0.1, **over)
    r = renderer_for(sc, "batched")
    render_scene(r, sc)
    assert_identical_to_oracle(r, sc)
