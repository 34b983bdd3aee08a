"""The canonical order where a bucket is too full to rank by counting (radix
passes instead, in the same scratch): keys of at most 32 bits and wider ones,
between frames sorted by buckets in one context (each clears its predecessor's
counts); and the numbers of roots on both sides of the lines where their starts
leave shared memory and where block sums are exchanged."""
import numpy as np
import pytest

from test_gpu_bns_stacks import _many_roots, _wall

pytestmark = pytest.mark.gpu

WINDOW = (1024, 768)
MAX_BUCKET = 2048     # mp_sort.cu, kMaxBucket


def _crowded(size, offset, culled=0):
    """A patch whose visible part lies about its parametric middle, where the
    paths of its four quarters are farthest apart, after `culled` patches behind
    the eye (more root bits)."""
    sc = _wall(size, *WINDOW)
    cp = sc.draws[0].mesh.cp
    cp[..., :2] += np.float32((offset - 0.0123) * size)
    behind = np.repeat(cp, culled, 0) * np.array([1, 1, -1], np.float32)
    sc.draws[0].mesh.cp = np.concatenate([behind, cp]).astype(np.float32)
    return sc


def _fullest_bucket(key):
    """Every root has as many buckets as sub-patches, spread over its path range by leading bits."""
    root, path = key >> np.uint64(32), (key & np.uint64(0xffffffff)).astype(np.int64)
    most = 0
    for r in np.unique(root):
        p = path[root == r]
        shift = max(0, int(p.max() - p.min()).bit_length() - (len(p).bit_length() - 1))
        most = max(most, int(np.bincount((p - p.min()) >> shift).max()))
    return most


def _key_bits(sc, rng):
    area = (rng[:, 2] - rng[:, 0]).astype(np.float64) * (rng[:, 3] - rng[:, 1])
    roots = sum(d.mesh.n_patches for d in sc.draws)
    return int(round(-np.log2(area.min()))) + (roots - 1).bit_length()


def _check(frames, opts, crowded):
    from micropolis_gb300.renderer import Projection, renderer_for
    from oracle import oracle
    r = renderer_for(frames[0], "batched", **opts)
    for k, sc in enumerate(frames):
        want = oracle.canonical_subpatches(sc, oracle.make_params(sc, **opts))
        if k in crowded:
            assert _fullest_bucket(want[3]) > MAX_BUCKET
            assert (_key_bits(sc, want[2]) > 32) == crowded[k]
        r.prepare()
        for d in sc.draws:
            r.load_patches(k, d.mesh.cp, d.mesh.type)
            r.draw_patches(k, d.mv, Projection(sc.fovy, sc.near, (sc.width, sc.height)), d.color)
        r.finish()
        for got, ref in zip(r.subpatches(), want[:3]):
            assert got.tobytes() == np.ascontiguousarray(ref, got.dtype).tobytes(), k
    r.close()


@pytest.mark.parametrize("wide", [False, True])
def test_crowded_bucket_between_others(built, cuda, wide):
    culled = 5000 if wide else 0
    frames = [_wall(1.5, *WINDOW), _crowded(256.0, 0.0, culled), _wall(3.0, *WINDOW), _crowded(256.0, 0.0001, culled),
              _crowded(64.0, 0.0, culled), _wall(1.5, *WINDOW)]
    _check(frames, dict(max_split_depth=31), {1: wide, 3: wide})   # (frame 4's fullest holds exactly MAX_BUCKET)


@pytest.mark.parametrize("roots", [8191, 8192, 8193, 12000, 16384, 16385])
def test_numbers_of_roots(built, cuda, roots):
    _check([_many_roots(roots)], {}, {})
