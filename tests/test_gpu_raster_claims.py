"""The fused kernel's blocks rasterize two groups of their own and claim the
others: lists of one sub-patch less and more than one, two and three groups
per resident block, drawn twice in one context (the claims start over each
frame), against the oracle at every pixel.  Patches of one sub-patch each lie
on a few thousand screen positions, equal ones on top of each other, so a
group taken twice or not at all changes a winner or the fragment count."""
import pytest

from helpers import assert_identical_to_oracle
from test_gpu_sort import _tiny

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dice, group, subs", [(8, 11, 14), (8, 8, 7), (16, 6, 5), (16, 2, 2)])
@pytest.mark.parametrize("rounds, more", [(1, -1), (1, 1), (2, 0), (2, 1), (3, -1), (3, 1)])
def test_every_group_once(built, cuda, dice, group, subs, rounds, more):
    import torch
    from micropolis_gb300.renderer import render_scene, renderer_for
    warps = 20   # per SM: 5 blocks of 128 threads or 10 of 64
    blocks = torch.cuda.get_device_properties(0).multi_processor_count * warps // (2 if subs in (7, 2) else 4)
    sc = _tiny(rounds * blocks * subs + more)
    sc.options["reyes_patch_size"] = dice
    r = renderer_for(sc, "batched", dice_group=group)
    for _ in range(2):
        render_scene(r, sc)
        assert r.stats()["subpatches"] == rounds * blocks * subs + more
    assert_identical_to_oracle(r, sc)
