"""Triangle kernels of the mixed preconditioner (two elements a warp, eight a
CTA): the scaled-face chain against the two-stage steps (DG_SCALED_FACES=0),
both FP32, 1e-4 of max |z| as for the other FP32 forms, and the FP32 apply
against the FP64 one, 1e-6 of max |y|.  Meshes of 2 to 98 triangles:
remainders 2, 0 and 2 of eight; vectors at 8-byte and at 4-byte boundaries."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def _at(v, off):
    buf = torch.empty(v.numel() + 2, dtype=v.dtype, device=v.device)
    buf[off:off + v.numel()] = v
    return buf[off:off + v.numel()]


@pytest.mark.parametrize("n", [1, 2, 4, 7])
@pytest.mark.parametrize("off", [0, 1])
def test_chain(n, off, monkeypatch):
    z = {}
    for scaled in ("0", "1"):
        monkeypatch.setenv("DG_SCALED_FACES", scaled)
        m = mesh.build_mesh("tri", n, seed=2)
        s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                     element.p3_element(m.ndim))
        s.build_operator()
        g = torch.Generator(device="cuda:0").manual_seed(3)
        r = torch.randn(s.nonods, dtype=torch.float32, device="cuda:0", generator=g)
        z[scaled] = s.precond_f32(_at(r, off), _at(torch.zeros_like(r), off)).clone()
        y = s.apply(r.double().contiguous())
        y32 = s.apply_f32(_at(r, off))
        assert float(torch.abs(y32.double() - y).max() / torch.abs(y).max()) < 1e-6
        s.close()
    assert float(torch.abs(z["0"] - z["1"]).max() / torch.abs(z["0"]).max()) < 1e-4
