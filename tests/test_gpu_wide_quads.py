"""Quads that cover many pixels: the wide raster (split limits above two pixels
a quad side) on both sides of the rule, with boxes from one pixel up to the
fast raster's largest, few subpixel bits (edges through pixel centres, where a
tie rule decides), quads of either winding, degenerate ones and quads that
leave the frame.  Batched frames equal the oracle's at every pixel, winners
included; the per-pass path and the overlapped launch its depth and fragments."""
import numpy as np
import pytest

from helpers import assert_identical_to_oracle

pytestmark = pytest.mark.gpu

W, H = 200, 136
PX = 2 * np.tan(np.radians(30.0)) / H           # a pixel at z = -1


def _scene(limit, **opts):
    """Bumpy patches facing the eye over windows from one pixel to beyond the
    frame, one turned around, one a point and one a line."""
    from micropolis_gb300 import scenes
    t = np.arange(4) / 3.0
    out = []
    boxes = [(5, 190, 4, 130), (-40, 60, -30, 70), (120, 260, 60, 200), (20, 33, 20, 29), (60, 61.2, 60, 61.1),
             (180, 90, 20, 100), (100, 164, 40, 104), (70, 70, 30, 30), (30, 150, 90, 90)]
    for k, (x0, x1, y0, y1) in enumerate(boxes):
        rng = np.random.default_rng(k)
        X, Y = np.meshgrid((x0 + (x1 - x0) * t - W / 2) * PX, (y0 + (y1 - y0) * t - H / 2) * PX)
        z = -1.0 - 0.05 * k + (0.15 if k < 7 else 0.0) * rng.uniform(-1, 1, size=(4, 4))
        cp = np.stack([X * -z, Y * -z, z], -1).reshape(1, 16, 3).astype(np.float32)
        mesh = scenes.Mesh(scenes.GREGORY, cp[:, scenes.BEZIER_TO_GREGORY]) if k % 3 == 2 else \
            scenes.Mesh(scenes.BEZIER, cp)
        out.append(scenes.Draw(mesh, np.eye(4, dtype=np.float32).reshape(16), (0.3 + 0.07 * k, 0.7, 0.5, 1.0)))
    return scenes.Scene("wide", W, H, out, options=dict(bound_n_split_limit=limit, **opts))


CASES = {
    "at_the_rule": dict(limit=16.0), "above_the_rule": dict(limit=16.5),
    "limit_24": dict(limit=24.0), "limit_40": dict(limit=40.0), "limit_100": dict(limit=100.0),
    "limit_128": dict(limit=128.0),
    "bits_1": dict(limit=40.0, subpixel_bits=1),
    "no_backface": dict(limit=50.0, backface_culling=0),
    "displaced": dict(limit=40.0, displacement=1, displacement_amplitude=0.5),
    "depth_cap": dict(limit=17.0, max_split_depth=3),
    "dice16_at": dict(limit=32.0, reyes_patch_size=16), "dice16_above": dict(limit=48.0, reyes_patch_size=16),
    "dice16_displaced": dict(limit=90.0, reyes_patch_size=16, displacement=1),
    "gpu_criterion": dict(limit=40.0, bound_criterion=1),
}


@pytest.mark.parametrize("name", list(CASES))
def test_frame_identical_to_oracle(built, cuda, name):
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    sc = _scene(**CASES[name])
    r = renderer_for(sc, "batched")
    render_scene(r, sc)
    stats = assert_identical_to_oracle(r, sc, oracle.make_params(sc))
    r.close()
    assert stats["fragments"] > 500
    depth = oracle.render(sc)[1]
    for path, over in (("plain", {}), ("batched", dict(overlap=1))):
        r = renderer_for(sc, path, **over)
        render_scene(r, sc)
        assert np.array_equal(r.read_framebuffer()[1], depth) and r.stats()["fragments"] == stats["fragments"], path
        r.close()


@pytest.mark.parametrize("group", [8, 16, 22])
def test_every_shape(built, cuda, group):
    from micropolis_gb300.renderer import render_scene, renderer_for
    sc = _scene(30.0)
    r = renderer_for(sc, "batched", dice_group=group)
    render_scene(r, sc)
    assert_identical_to_oracle(r, sc)
    r.close()
