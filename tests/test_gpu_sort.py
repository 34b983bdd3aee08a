"""The canonical order's bucket sort at its edges: none to a handful of
sub-patches, counts on both sides of a block's threads, keys with more bits
than buckets, buckets too full to rank by counting and keys too wide for it
(radix passes instead), and frames of different sizes after one another in
one context (each clears its predecessor's counts)."""
import numpy as np
import pytest

from test_gpu_bns_stacks import _many_roots, _wall

pytestmark = pytest.mark.gpu


def _tiny(n):
    """n patches of one sub-patch each, in reverse screen order."""
    from micropolis_gb300 import scenes
    t = (np.arange(4) / 3.0 - 0.5) * 0.005
    X, Y = np.meshgrid(t, t)
    k = np.arange(n)[::-1]
    off = np.stack([(k % 64) * 0.016 - 0.5, (k // 64 % 48) * 0.016 - 0.4, 0 * k], -1)
    cp = np.stack([X, Y, -1.0 + 0 * X], -1).reshape(1, 16, 3) + off[:, None]
    return scenes.Scene("tiny", 512, 384, [scenes.Draw(scenes.Mesh(scenes.BEZIER, cp.astype(np.float32)),
                                                       np.eye(4, dtype=np.float32).reshape(16))])


def _wide(culled, size):
    """A deeply split patch after `culled` patches behind the eye, in a small
    frame: more key bits than 32 above the bucket's."""
    sc = _wall(size, 64, 48)
    cp = sc.draws[0].mesh.cp
    behind = np.repeat(cp, culled, 0) * np.array([1, 1, -1], np.float32)
    sc.draws[0].mesh.cp = np.concatenate([behind, cp])
    return sc


CASES = [("tiny_0", lambda: [_tiny(0)]), ("tiny_1", lambda: [_tiny(1)]), ("tiny_2", lambda: [_tiny(2)]),
         ("tiny_3", lambda: [_tiny(3)]), ("tiny_5", lambda: [_tiny(5)]), ("tiny_511", lambda: [_tiny(511)]),
         ("tiny_513", lambda: [_tiny(513)]), ("tiny_3000", lambda: [_tiny(3000)]),
         ("one_bucket", lambda: [_wall(256.0)]), ("wide_keys", lambda: [_wide(5000, 8192.0)]),
         ("many_roots", lambda: [_many_roots(30001)]),
         ("in_turn", lambda: [_wall(1.5), _tiny(7), _wall(256.0), _tiny(3000), _tiny(0), _wall(1.5), _wall(3.0)])]


@pytest.mark.parametrize("name", [n for n, _ in CASES])
def test_canonical_order(built, cuda, name):
    from micropolis_gb300.renderer import Projection, renderer_for
    from oracle import oracle
    frames = dict(CASES)[name]()
    opts = dict(max_split_depth=31)
    r = renderer_for(frames[0], "batched", **opts)
    for k, sc in enumerate(frames):
        want = oracle.canonical_subpatches(sc, oracle.make_params(sc, **opts))
        r.prepare()
        for d in sc.draws:
            r.load_patches(k, d.mesh.cp, d.mesh.type)
            r.draw_patches(k, d.mv, Projection(sc.fovy, sc.near, (sc.width, sc.height)), d.color)
        r.finish()
        for got, ref in zip(r.subpatches(), want):
            assert got.tobytes() == np.ascontiguousarray(ref, got.dtype).tobytes(), (name, k)
    r.close()
