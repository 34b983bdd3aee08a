"""Frames of different numbers of draws in one context: the list of each is the
oracle's, and a small frame costs the same after a large one as before it."""
import numpy as np
import pytest

from test_gpu_bns_stacks import _draws

pytestmark = pytest.mark.gpu


def test_draw_counts_in_turn(built, cuda):
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    scenes = {n: _draws(n) for n in (1, 40, 3, 9, 0)}
    r = renderer_for(scenes[1], "batched")
    for n in (1, 40, 3, 9, 0, 40, 1):
        render_scene(r, scenes[n])
        want = oracle.canonical_subpatches(scenes[n], oracle.make_params(scenes[n]))
        for got, ref in zip(r.subpatches(), want):
            assert got.tobytes() == np.ascontiguousarray(ref, got.dtype).tobytes(), n
    r.close()


def test_small_frame_after_a_large_one(built, cuda):
    """(a frame that uploads the records of 40,000 draws takes more than twice as long)"""
    from micropolis_gb300.renderer import Projection, render_scene, renderer_for
    sc = _draws(1)
    r = renderer_for(sc, "batched")
    proj = Projection(sc.fovy, sc.near, (sc.width, sc.height))

    def gpu_ms(frames=40):
        out = []
        for _ in range(frames):
            render_scene(r, sc)
            out.append(r.stats()["gpu_ms"])
        return float(np.median(out))

    before = gpu_ms()
    r.load_patches(7, sc.draws[0].mesh.cp[:1], sc.draws[0].mesh.type)
    away = np.eye(4, dtype=np.float32)
    away[3, 2] = 1000.0                  # behind the eye: nothing to draw
    r.prepare()
    for _ in range(40000):
        r.draw_patches(7, away, proj)
    r.finish()
    after = gpu_ms()
    r.close()
    assert after < 1.5 * before, (before, after)
