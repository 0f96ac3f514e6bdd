"""The estimate of lambda_max(A_ee^-1 A) behind the mixed preconditioner's
Chebyshev schedule does not depend on the smoother's weight w, though the
power iteration runs on w A_ee^-1 A: w of 1e-3 to 2 give the estimate of the
default 0.8 to twice the iteration's stopping tolerance (1e-3), with scaled
faces (BF16 on tetrahedra, FP32 on triangles) and without."""
import re

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("kind,n,faces", [("tet", 4, "1"), ("tet", 4, "0"), ("tri", 8, "1"), ("tri", 8, "0")])
def test_estimate_independent_of_the_weight(kind, n, faces, monkeypatch, capfd):
    monkeypatch.setenv("DG_VERBOSE", "1")
    monkeypatch.setenv("DG_SCALED_FACES", faces)
    m = mesh.build_mesh(kind, n, seed=4)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.build_operator()
    b = s.rhs(torch.ones(s.nonods, dtype=torch.float64, device="cuda:0"))
    est = {}
    for w in (0.8, 1e-3, 0.02, 2.0):
        s.set_mixed_options(smooth_w=w)
        capfd.readouterr()
        s.solve_mixed(torch.zeros_like(b), b, 0.5 * float(torch.linalg.norm(b)))
        out = re.findall(r"lambda_max\(A_ee\^-1 A\) ~ ([0-9.]+)", capfd.readouterr().err)
        assert len(out) == 1, (w, out)
        est[w] = float(out[0])
    print(kind, n, faces, est)
    assert all(abs(v / est[0.8] - 1) <= 2e-3 for v in est.values()), est
    s.close()
