"""The overlapped launch, whose bound-and-split blocks rasterize afterwards out
of the shared memory that held their rings: frames of every block shape, with
displacement, more draws than are staged, and a bundle queue without room
(pairs stay on the small rings until they are full, then the frame regrows).
Sub-patches equal the oracle's as sets, ranges bounded, fragments and every
pixel's depth exactly (which of two equally deep micropolygons wins follows
the emission order)."""
import numpy as np
import pytest

from test_gpu_bns_stacks import _draws, _wall

pytestmark = pytest.mark.gpu

CASES = {
    "group_8": (lambda: _draws(9), dict(dice_group=8)),
    "group_11": (lambda: _draws(8), dict(dice_group=11)),
    "group_16": (lambda: _draws(9), dict(dice_group=16, displacement=1)),
    "group_22": (lambda: _wall(1.5, patches=20), dict(dice_group=22)),
    "dice16_group_2": (lambda: _draws(5), dict(reyes_patch_size=16, dice_group=2)),
    "dice16_group_6": (lambda: _draws(5), dict(reyes_patch_size=16, displacement=1)),
    "one_bns_block": (lambda: _draws(5), dict(bns_blocks=1)),
    "no_queue": (lambda: _wall(1.5, 1024, 768), dict(queue_capacity=1)),
    "no_queue_many": (lambda: _wall(1.5, patches=20), dict(queue_capacity=1)),
}


def _bits(draw, pid, rng):
    return sorted(zip(np.asarray(draw).tolist(), np.asarray(pid).tolist(),
                      map(bytes, np.ascontiguousarray(rng, np.float32))))


@pytest.mark.parametrize("name", list(CASES))
def test_overlapped_frame(built, cuda, name):
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    make, over = CASES[name]
    sc = make()
    shape = {k: v for k, v in over.items() if k in ("reyes_patch_size", "displacement")}
    p = oracle.make_params(sc, **shape)
    draw, pid, rng, *_ = oracle.canonical_subpatches(sc, p)
    bounds = sum(oracle.bound_n_split(sc, k, p)[2] for k in range(len(sc.draws)))
    _, depth, stats = oracle.render(sc, params=p)
    r = renderer_for(sc, "batched", overlap=1, **over)
    for _ in range(3):
        render_scene(r, sc)
        assert _bits(*r.subpatches()) == _bits(draw, pid, rng)
        assert r.stats()["bounds"] == bounds and r.stats()["fragments"] == stats["fragments"]
        assert np.array_equal(r.read_framebuffer()[1], depth)
    r.close()
