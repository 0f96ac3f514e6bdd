"""The batched solve times the smoothing variants only where it would run the
fastest: not on the scaled faces, whose solve then holds none of their layouts;
where it is asked to (once); and without scaled faces once per build."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("faces", ["1", "0"])
def test_variants_timed_where_they_run(faces, monkeypatch):
    monkeypatch.setenv("DG_SCALED_FACES", faces)
    m = mesh.build_mesh("tet", 4, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(3))
    s.build_operator()
    b = s.rhs(torch.ones(s.nonods, dtype=torch.float64, device="cuda:0"))
    B = torch.stack([b, 2.0 * b])
    tol = 1e-9 * float(torch.linalg.norm(b))

    def solve():
        X = torch.zeros_like(B)
        s.solve_mixed_batched(X, B, tol, raise_noconv=True)
        return X

    X = solve()
    chosen, us = s.batched_tuning()
    assert (not us and chosen == "mma_sync4") if faces == "1" else us[chosen] == min(us.values())
    held = s.info()["device_bytes"]
    s.set_batched_kernel("auto")
    assert float((solve() - X).abs().max()) <= 1e-6 * float(X.abs().max())
    chosen, us = s.batched_tuning()
    assert len(us) == 7 and us[chosen] == min(us.values())
    # the tensor-core layout and two split iterates, 5,760 + 2 x 6,144 bytes an element
    assert s.info()["device_bytes"] - held >= (m.nele * 18048 if faces == "1" else 0)
    s.build_operator()
    solve()
    again = s.batched_tuning()[1]
    assert (again == us) == (faces == "1")
    s.close()
