"""FP32 Gram-Schmidt of the mixed solve where the update adds the block sums
of the dots itself (up to 128 blocks), where the scaling adds those of the
norm (up to 256), and above: 2 to 322 blocks, restart lengths on both sides of
32 vectors.  The FP64 residual meets the solve's tolerance, and the iteration
counts of the restart lengths that hold the whole inner solve agree."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("kind,n", [("tri", 10), ("tet", 8), ("tet", 10), ("tet", 11), ("tet", 13), ("tet", 14)])
def test_block_sums(kind, n):
    m = mesh.build_mesh(kind, n, seed=4)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.build_operator()
    g = torch.Generator(device="cuda:0").manual_seed(3)
    b = s.rhs(torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g))
    tol = 1e-10 * float(torch.linalg.norm(b))
    its = []
    for restart in (5, 31, 40):
        x = torch.zeros_like(b)
        out = s.solve_mixed(x, b, tol, m=restart)
        assert float(torch.linalg.norm(s.residual(x, b))) <= tol * (1 + 1e-9)
        its.append(out[0])
    assert its[1] == its[2]
    s.close()
