"""FP64 V-cycle with its coarse tail as one matrix, and the FP64 Gram-Schmidt
kernels, at the sizes where they can go wrong.

V-cycle: dg_mg_vcycle against the CPU restatement, the parity tests'
tolerance (1e-12 of the largest entry) over meshes whose whole V-cycle is
the matrix (even and odd row counts, one to a few rows), and with the matrix
starting below level 0 (DG_TAIL_MAX64), with V(3,3), V(2,2), V(1,0).

Gram-Schmidt: GMRES with restart lengths over the kernels' groups (8 vectors
a row, 32 a pass; partial sums added in the update or apart) solves the same
system; the solutions agree to the solve's own accuracy."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402
from oracle.dg_oracle import OracleDG  # noqa: E402


@pytest.mark.parametrize("kind,n,pre,post,rows", [("tri", 1, 3, 3, ""), ("tri", 3, 2, 2, ""), ("tri", 6, 3, 3, ""),
                                                  ("tri", 9, 2, 2, "20"), ("tet", 3, 1, 0, "9"), ("tet", 4, 2, 2, "1"),
                                                  ("tet", 4, 3, 3, "40")])
def test_vcycle_tail_matrix(kind, n, pre, post, rows, monkeypatch):
    if rows:
        monkeypatch.setenv("DG_TAIL_MAX64", rows)
    m = mesh.build_mesh(kind, n, seed=4)
    el = element.p3_element(m.ndim)
    order = sfc.hilbert_sfc_order(m.cg_coords)
    s = DGSolver(m, order, SolverConfig(pre_smooth_its=pre, post_smooth_its=post), el)
    s.build_operator()
    O = OracleDG(m, el, element.drst_duv(m.ndim), pre_smooth_its=pre, post_smooth_its=post)
    ctx = O.setup(order)
    r = np.random.default_rng(5).standard_normal(m.cg_nonods)
    for _ in range(2):
        e = s.mg_vcycle(torch.tensor(r, device="cuda:0")).cpu().numpy()
        ref = O.mg_on_p1cg(r, ctx["levels"], ctx["sizes"])
        assert np.abs(e - ref).max() <= 1e-12 * np.abs(ref).max()
    s.close()


@pytest.mark.parametrize("kind,n", [("tri", 8), ("tet", 8)])
def test_gram_schmidt_groups(kind, n):
    m = mesh.build_mesh(kind, n, seed=4)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.build_operator()
    g = torch.Generator(device="cuda:0").manual_seed(3)
    b = s.rhs(torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g))
    tol = 1e-11 * float(torch.linalg.norm(b))
    xs = []
    for restart in (7, 8, 9, 33, 40):
        x = torch.zeros_like(b)
        _, res = s.gmres(x, b, tol, m=restart, max_its=4000, raise_noconv=True)
        assert float(torch.linalg.norm(s.residual(x, b))) <= tol * (1 + 1e-9)
        xs.append(x)
    for x in xs[1:]:
        assert float(torch.abs(x - xs[0]).max() / torch.abs(xs[0]).max()) < 1e-8
    s.close()
