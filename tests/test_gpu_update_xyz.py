"""Control points updated from xyz triples in device memory: the frame equals
the one of a fresh upload, at point counts around a block of threads, and
mistakes are status codes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,gregory", [(1, False), (15, True), (16, False), (17, False), (333, True)])
def test_update_equals_upload(built, cuda, n, gregory):
    torch = cuda
    from micropolis_gb300 import _lib, scenes
    from micropolis_gb300.renderer import render_scene, renderer_for
    mv = scenes.look_at((8, -11, 5), (0, 0, 0), (0, 0, 1))
    a, b = (scenes.scattered_patches(np.random.default_rng(s), n, gregory) for s in (1, 2))
    frames = []
    for mesh, update in ((b, None), (a, b)):
        sc = scenes.Scene("update", 320, 240, [scenes.Draw(mesh, mv)])
        r = renderer_for(sc, "batched")
        r.load_patches(1, mesh.cp, mesh.type)
        if update is not None:
            with pytest.raises(_lib.MpError):
                r.update_patches_xyz_device(2, 16)   # an unknown handle: refused before the address is used
            with pytest.raises(_lib.MpError):
                r.update_patches_xyz_device(1, 0)
            xyz = torch.tensor(update.cp, device="cuda")
            torch.cuda.synchronize()
            r.update_patches_xyz_device(1, xyz.data_ptr())
        render_scene(r, sc, [1])
        frames.append((*r.subpatches(), *r.read_framebuffer(), r.visibility()))
        r.close()
    for x, y in zip(*frames):
        assert x.tobytes() == y.tobytes()
