"""adjoint.backward_work counts the updates that the adjoint issues: one per
control-point coordinate and distinct patch of each warp of 32 pixels."""
import numpy as np

from micropolis_gb300 import adjoint, scenes


class _Frame:
    class options:
        reyes_patch_size = 8

    def __init__(self, vis, draw, pid):
        self.vis, self.list = vis, (draw, pid, None)

    def visibility(self, view):
        return self.vis

    def subpatches(self):
        return self.list


def test_updates_per_distinct_patch_of_a_warp():
    rng = np.random.default_rng(0)
    meshes = [scenes.scattered_patches(rng, 5, False), scenes.scattered_patches(rng, 3, True)]
    sc = scenes.Scene("two", 64, 32, [scenes.Draw(m, np.eye(4, dtype=np.float32).reshape(16)) for m in meshes])
    draw = rng.integers(0, 2, 40).astype(np.int32)
    pid = (rng.integers(0, 1 << 20, 40) % np.where(draw == 0, 5, 3)).astype(np.int32)
    vis = np.where(rng.random(64 * 32) < 0.7, rng.integers(0, 40 * 64, 64 * 32), -1)
    vis[:32] = 7            # a warp that sees one patch
    vis[32:64] = -1         # and one that sees none
    want = 0
    for warp in vis.reshape(-1, 32):
        seen = {(draw[v // 64], pid[v // 64]) for v in warp if v >= 0}
        want += sum(3 * (16, 20)[d] for d, _ in seen)
    work = adjoint.backward_work(sc, _Frame(vis, draw, pid))
    assert work["A_bwd"] == want and work["covered_pixels"] == int((vis >= 0).sum())
    empty = adjoint.backward_work(sc, _Frame(np.full(64 * 32, -1), draw[:0], pid[:0]))
    assert empty["A_bwd"] == 0 and empty["covered_pixels"] == 0
