"""Level values whose summation lists are long (a warp an entry above 64, a
CTA above 1,024 Galerkin values): the FP64 V-cycle of a first build and of a
rebuild against the CPU restatement, the parity tests' tolerance (1e-12 of the
largest entry).  16 to 441 vertices: longest lists of about a hundred values, a
few hundred, and above 1,024 with levels of each kind."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402
from oracle.dg_oracle import OracleDG  # noqa: E402


@pytest.mark.parametrize("kind,n", [("tri", 3), ("tri", 8), ("tri", 20), ("tet", 2), ("tet", 5)])
def test_long_level_sums(kind, n):
    m = mesh.build_mesh(kind, n, seed=4)
    el = element.p3_element(m.ndim)
    order = sfc.hilbert_sfc_order(m.cg_coords)
    s = DGSolver(m, order, SolverConfig(pre_smooth_its=2, post_smooth_its=2), el)
    O = OracleDG(m, el, element.drst_duv(m.ndim), pre_smooth_its=2, post_smooth_its=2)
    ctx = O.setup(order)
    r = np.random.default_rng(5).standard_normal(m.cg_nonods)
    ref = O.mg_on_p1cg(r, ctx["levels"], ctx["sizes"])
    for _ in range(2):
        s.build_operator()
        e = s.mg_vcycle(torch.tensor(r, device="cuda:0")).cpu().numpy()
        assert np.abs(e - ref).max() <= 1e-12 * np.abs(ref).max()
    s.close()
