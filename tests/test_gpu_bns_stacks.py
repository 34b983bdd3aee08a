"""Bound-and-split's per-warp stacks and hand-over at the sizes where they
change course: one root whose tree feeds the whole grid, more roots than the
grid holds at once (the rest is dealt with atomics), trees deeper than the
exact-sample depth, more draws than are staged in shared memory, a queue
without room (pairs stay, or the frame regrows), and the overlapped kernel's
small rings.  Sub-patch lists equal the oracle's canonical list bit for bit,
and the number of bounded ranges equals the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wall(size, width=512, height=384, patches=1):
    """Nearly flat patches facing the eye one unit away, `size` wide: only the
    visible part is split, to depth 2 log2(size * width / 9)."""
    from micropolis_gb300 import scenes
    t = (np.linspace(-0.5, 0.5, 4) + 0.0123) * size
    X, Y = np.meshgrid(t, t)
    cp = np.stack([X, Y, -1.0 - 0.01 * np.sin(np.arange(16.0)).reshape(4, 4)], -1).reshape(1, 16, 3)
    cp = np.repeat(cp, patches, 0).astype(np.float32)
    return scenes.Scene("wall", width, height,
                        [scenes.Draw(scenes.Mesh(scenes.BEZIER, cp), np.eye(4, dtype=np.float32).reshape(16))])


def _many_roots(n):
    from micropolis_gb300 import scenes
    rng = np.random.default_rng(5)
    m = scenes.scattered_patches(rng, n, gregory=False)
    m.cp[:] = m.cp.mean(1, keepdims=True) + 0.05 * (m.cp - m.cp.mean(1, keepdims=True))
    return scenes.Scene("roots", 256, 192, [scenes.Draw(m, scenes.look_at((8, -11, 5), (0, 0, 0), (0, 0, 1)))])


def _draws(n):
    from micropolis_gb300 import scenes
    rng = np.random.default_rng(6)
    mv = scenes.look_at((8, -11, 5), (0, 0, 0), (0, 0, 1))
    return scenes.Scene("draws", 320, 240, [scenes.Draw(scenes.scattered_patches(rng, 3, k % 2 == 1), mv)
                                            for k in range(n)])


CASES = {
    "one_root": (lambda: _wall(1.5, 1024, 768), {}),
    "deep": (lambda: _wall(256.0), dict(max_split_depth=60)),
    "deep_gpu_criterion": (lambda: _wall(256.0), dict(max_split_depth=60, bound_criterion=1)),
    "roots_100001": (lambda: _many_roots(100001), {}),
    "draws_8": (lambda: _draws(8), {}),
    "draws_9": (lambda: _draws(9), {}),
    "no_queue": (lambda: _wall(1.5, 1024, 768), dict(queue_capacity=1)),
    "overlap": (lambda: _wall(1.5, patches=20), dict(overlap=1)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_subpatches_match_oracle(built, cuda, name):
    from micropolis_gb300.renderer import render_scene, renderer_for
    from oracle import oracle
    make, over = CASES[name]
    sc = make()
    p = oracle.make_params(sc, **{k: v for k, v in over.items() if k in ("max_split_depth", "bound_criterion")})
    draw, pid, rng, *_ = oracle.canonical_subpatches(sc, p)
    bounds = sum(oracle.bound_n_split(sc, k, p)[2] for k in range(len(sc.draws)))
    r = renderer_for(sc, "batched", **over)
    for _ in range(2):
        render_scene(r, sc)
        gd, gp, gr = r.subpatches()
        if over.get("overlap"):
            # the overlapped kernel keeps emission order: compare as sets
            bits = lambda d, q, g: sorted(zip(d.tolist(), q.tolist(), map(bytes, np.ascontiguousarray(g, np.float32))))
            assert bits(gd, gp, gr) == bits(np.asarray(draw), np.asarray(pid), np.asarray(rng))
        else:
            assert np.array_equal(gd, draw) and np.array_equal(gp, pid)
            assert np.array_equal(gr.view(np.uint32), np.ascontiguousarray(rng, np.float32).view(np.uint32))
        assert r.stats()["bounds"] == bounds
    r.close()
    if name == "deep":
        assert ((rng[:, 2] - rng[:, 0]) * (rng[:, 3] - rng[:, 1])).min() < 2.0 ** -24
