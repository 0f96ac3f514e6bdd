"""FP32 Gram-Schmidt with more than 32 basis vectors, where the dots run in two
passes and the update no longer adds their block sums itself: inner cycles of
over 32 steps (one smoothing step per leg, inner tolerance 1e-6, restart 80;
the steps of each refinement step from the verbose trace) on both sides of 128
and 256 block sums.  The FP64 residual meets the tolerance, and the solution
agrees with restart 31 and with FP64 GMRES to what a residual of 1e-10 leaves
(1e-7, as the mixed tests)."""
import re

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("passes", ["1", "2"])
@pytest.mark.parametrize("kind,n", [("tri", 40), ("tet", 8), ("tet", 12), ("tet", 14)])
def test_more_than_32_vectors(kind, n, passes, monkeypatch, capfd):
    monkeypatch.setenv("DG_MIXED_SWEEPS", "1")
    monkeypatch.setenv("DG_MIXED_CGS", passes)
    monkeypatch.setenv("DG_VERBOSE", "1")
    m = mesh.build_mesh(kind, n, seed=4)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.set_mixed_options(smoother="jacobi3" if kind == "tri" else "blockinv")
    s.build_operator()
    g = torch.Generator(device="cuda:0").manual_seed(3)
    b = s.rhs(torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g))
    tol = 1e-10 * float(torch.linalg.norm(b))
    ref = torch.zeros_like(b)
    s.gmres(ref, b, tol, raise_noconv=True, max_its=4000)
    for restart in (31, 80):
        x = torch.zeros_like(b)
        capfd.readouterr()
        s.solve_mixed(x, b, tol, m=restart, inner_rtol=1e-6, raise_noconv=True)
        total = [0] + [int(k) for k in re.findall(r"inner its total (\d+)", capfd.readouterr().err)]
        steps = [j - i for i, j in zip(total, total[1:])]
        print(kind, n, passes, restart, steps)
        if restart == 80:
            assert 32 < max(steps) <= 80
        assert float(torch.linalg.norm(s.residual(x, b))) <= tol * (1 + 1e-9)
        assert float((x - ref).abs().max()) <= 1e-7 * float(ref.abs().max())
    s.close()
