"""DiffRenderer.render refuses control points of too few patches."""
import pytest

from test_gpu_adjoint_groups import _grid

pytestmark = pytest.mark.gpu


def test_too_few_control_points(built, cuda):
    torch = cuda
    from micropolis_gb300 import adjoint
    sc = _grid(2, 2)
    dr = adjoint.DiffRenderer(sc)
    cp = torch.tensor(sc.draws[0].mesh.cp, device="cuda")
    want = dr.render(cp, 1.0)
    with pytest.raises(ValueError):
        dr.render(cp[:3], 1.0)
    assert torch.equal(dr.render(cp, 1.0), want)     # the refused call left nothing behind
    dr.r.close()
