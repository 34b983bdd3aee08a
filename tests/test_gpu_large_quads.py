"""Quads too large for the fast raster: more of them than the first list holds
(the status is set while the fused kernel runs, then the frame regrows), and
their number, the same on both paths."""
import numpy as np
import pytest

from helpers import assert_identical_to_oracle

pytestmark = pytest.mark.gpu

W, H = 192, 128
PX = 2 * np.tan(np.radians(30.0)) / H           # a pixel at z = -1


def _walls(n):
    """n patches facing the eye, each one sub-patch of 64 quads of 25 by 17 pixels, the last ones nearest."""
    from micropolis_gb300 import scenes
    t = np.linspace(-0.52, 0.52, 4)
    X, Y = np.meshgrid(W * PX * t, H * PX * t)
    z = -1.0 - 1e-5 * np.arange(n)[::-1, None]
    cp = np.stack([X.ravel() * -z, Y.ravel() * -z, np.repeat(z, 16, 1)], -1).astype(np.float32)
    return scenes.Scene("walls", W, H, [scenes.Draw(scenes.Mesh(scenes.BEZIER, cp),
                                                    np.eye(4, dtype=np.float32).reshape(16))],
                        options=dict(bound_n_split_limit=400.0))


@pytest.mark.parametrize("n", [1025, 2500])
def test_list_overflows_while_rasterizing(built, cuda, n):
    from micropolis_gb300.renderer import render_scene, renderer_for
    sc = _walls(n)
    assert n * 64 > 1 << 16
    r = renderer_for(sc, "batched")
    for _ in range(2):
        render_scene(r, sc)
        assert_identical_to_oracle(r, sc)
    r.close()


@pytest.mark.parametrize("dice, limit, culling", [(8, 100.0, 1), (8, 200.0, 1), (8, 200.0, 0), (16, 300.0, 1)])
def test_number_of_large_quads(built, cuda, dice, limit, culling):
    """(blocks without a front-facing quad hold some that have no tile to visit)"""
    from micropolis_gb300 import scenes
    from micropolis_gb300.renderer import render_scene, renderer_for
    rng = np.random.default_rng(3)
    mv = scenes.look_at((8, -11, 5), (0, 0, 0), (0, 0, 1))
    sc = scenes.Scene("mixed", 1920, 1080, [scenes.Draw(scenes.scattered_patches(rng, 700, g), mv) for g in (False, True)],
                      options=dict(reyes_patch_size=dice, bound_n_split_limit=limit, backface_culling=culling))
    count = []
    for path in ("plain", "batched"):
        r = renderer_for(sc, path)
        render_scene(r, sc)
        count.append(r.stats()["big_quads"])
        r.close()
    assert count[0] == count[1] > 0
