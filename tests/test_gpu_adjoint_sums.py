"""The sum of a warp's values where all of its pixels see one patch: within the
bound of pairwise summation, log2(32) half-ulps of the magnitudes' sum, also
when one value is so large that each other one added to it by itself is lost.
Every lane's own value is known exactly: a gradient image with that pixel alone
adds it to zero."""
import numpy as np
import pytest

from test_gpu_adjoint_groups import H, W, _grid

pytestmark = pytest.mark.gpu

FIRST = (W // 8 * 6 + 8) * 64     # 32 pixels in the middle of the frame: half an 8x8 tile, one warp


@pytest.mark.parametrize("gregory", [False, True])
def test_warp_sum_is_pairwise(built, cuda, gregory):
    torch = cuda
    from micropolis_gb300 import adjoint
    sc = _grid(1, 1, gregory)
    dr = adjoint.DiffRenderer(sc)
    cp = torch.tensor(sc.draws[0].mesh.cp, device="cuda")
    dr.render(cp, 1.0)
    assert (dr.r.visibility(0)[FIRST:FIRST + 32] >= 0).all()

    def gradient(weights):
        g = torch.zeros((W * H, 4), device="cuda")
        g[FIRST:FIRST + 32, 0] = torch.tensor(weights, dtype=torch.float32, device="cuda")
        out, _ = dr.backward(g, tuple(cp.shape), cp.device)
        torch.cuda.synchronize()
        return out.double().cpu().numpy().ravel()

    eye = np.eye(32)
    alone = np.array([gradient(e) for e in eye])
    for big in (0, 13, 31):
        # the others at 0.4 ulp of the big lane's largest coordinate, of its sign
        j = np.abs(alone[big]).argmax()
        ulp = float(np.spacing(np.float32(abs(alone[big, j]))))
        w = 0.4 * ulp * np.sign(alone[big, j]) / alone[:, j]
        w[big] = 1.0
        values = np.array([gradient(w[k] * eye[k]) for k in range(32)])
        total = gradient(w)
        bound = 5 * 2.0 ** -24 * np.abs(values).sum(0)
        assert (np.abs(total - values.sum(0)) <= bound).all(), big
        assert np.abs(np.delete(values, big, 0)[:, j]).sum() > 12 * ulp     # lost one by one
    dr.r.close()
