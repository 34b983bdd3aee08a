"""The displacement of dice vertices at the edges of its sine's range: the
short form (arguments below 2^22 pi, positions within 2^18 of the eye's axes)
and the general one give the oracle's floats bit for bit, infinities and NaN
included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _far_scene(scale, amplitude, nan=False):
    """Patches behind the eye (culled whole, so the frame is empty) whose x
    and y reach +-scale; their vertices are diced through the debug entry."""
    from micropolis_gb300 import scenes
    rng = np.random.default_rng(11)
    cp = rng.uniform(-1, 1, size=(8, 16, 3)) * np.array([scale, scale, 1.0]) + np.array([0.0, 0.0, 5.0])
    cp = cp.astype(np.float32)
    if nan:
        cp[0, 3, 0] = np.nan
        cp[1, 7, 1] = np.inf
    d = scenes.Draw(scenes.Mesh(scenes.BEZIER, cp), np.eye(4, dtype=np.float32).reshape(16))
    return scenes.Scene("far", 256, 192, [d], options=dict(displacement=1, displacement_amplitude=amplitude))


@pytest.mark.parametrize("scale,amplitude,nan", [(1e-30, 1.0, False), (1.0, 1.0, False), (1.0, 0.0, False),
                                                 (262143.0, 1.0, False), (262145.0, 1.0, False),
                                                 (300000.0, -1.0, False), (1e8, 1.0, False), (1.0, 1e7, False),
                                                 (1.0, 1.0, True)])
def test_displaced_vertices_match_oracle(built, cuda, scale, amplitude, nan):
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    sc = _far_scene(scale, amplitude, nan)
    r = renderer_for(sc, "batched")
    render_scene(r, sc)
    pid = np.arange(8, dtype=np.int32)
    rng = np.tile(np.array([[0, 0, 1, 1]], np.float32), (8, 1))
    pos, _, _ = r.dice_subpatches(0, pid, rng)
    r.close()
    for k in range(8):
        want, _, _ = oracle.dice(sc, 0, pid[k], rng[k])
        assert np.array_equal(pos[k], want, equal_nan=True), (k, np.count_nonzero(pos[k] != want))
