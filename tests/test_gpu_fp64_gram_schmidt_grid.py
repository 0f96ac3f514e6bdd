"""FP64 Gram-Schmidt where the update changes its CTA size (64 threads up to
64 x 2 SMs entry pairs) and the dots their share of a thread (one entry pair
up to 16,384): the stored basis of short restarts solves the same system as
the longest one, residual and solution to the solve's own accuracy."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("kind,n", [("tri", 1), ("tri", 40), ("tri", 41), ("tri", 44), ("tri", 45)])
def test_update_grid(kind, n):
    m = mesh.build_mesh(kind, n, seed=4)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.build_operator()
    g = torch.Generator(device="cuda:0").manual_seed(3)
    b = s.rhs(torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g))
    tol = 1e-11 * float(torch.linalg.norm(b))
    xs = []
    for restart in (9, 32, 40):
        x = torch.zeros_like(b)
        s.gmres(x, b, tol, m=restart, max_its=4000, raise_noconv=True)
        assert float(torch.linalg.norm(s.residual(x, b))) <= tol * (1 + 1e-9)
        xs.append(x)
    for x in xs[1:]:
        assert float(torch.abs(x - xs[0]).max() / torch.abs(xs[0]).max()) < 1e-8
    s.close()
