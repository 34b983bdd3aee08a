"""Bound-and-split with fewer and with more blocks than the device holds at once
(those that do not fit start only when others end): the same list, bit for
bit, for one root whose tree feeds the whole launch, more roots than shares,
and roots in many draws."""
import numpy as np
import pytest

from test_gpu_bns_stacks import _draws, _many_roots, _wall

pytestmark = pytest.mark.gpu

SCENES = {
    "one_root": lambda: _wall(1.5, 1024, 768),
    "roots_700": lambda: _many_roots(700),
    "roots_100001": lambda: _many_roots(100001),
    "draws_9": lambda: _draws(9),
}


@pytest.mark.parametrize("criterion", [0, 1])
@pytest.mark.parametrize("name", list(SCENES))
def test_any_number_of_blocks(built, cuda, name, criterion):
    import torch
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    sc = SCENES[name]()
    draw, pid, rng, *_ = oracle.canonical_subpatches(sc, oracle.make_params(sc, bound_criterion=criterion))
    r = renderer_for(sc, "batched", bound_criterion=criterion)
    fits = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    for blocks in (1, 3, fits - 1, fits + 1, 3 * fits, 0):
        r.set_bns_blocks(blocks)
        for _ in range(2):
            render_scene(r, sc)
            gd, gp, gr = r.subpatches()
            assert np.array_equal(gd, draw) and np.array_equal(gp, pid), blocks
            assert np.array_equal(gr.view(np.uint32), np.ascontiguousarray(rng, np.float32).view(np.uint32)), blocks
    r.close()


def test_refused_counts(built, cuda):
    from micropolis_gb300._lib import MpError
    from micropolis_gb300.renderer import renderer_for
    r = renderer_for(_draws(1), "batched")
    for blocks in (-1, 65536):
        with pytest.raises(MpError):
            r.set_bns_blocks(blocks)
    r.close()
