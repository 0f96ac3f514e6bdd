"""The digit copy of the blocks is given back when another buffer does not fit:
with the device memory of a context limited (DG_MEM_LIMIT) to less than what
it takes with the digits but enough without, FP64, mixed and batched solves
run as before and the digits are gone; with too little for what a solve must
have, the allocation error stays."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300._capi import DGError  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def _run(mode, limit, monkeypatch):
    monkeypatch.setenv("DG_MEM_LIMIT", str(limit))
    m = mesh.build_mesh("tet", 4, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(3))
    s.set_build_mode(mode)
    held = []
    try:
        s.build_operator()
        b = s.rhs(torch.ones(s.nonods, dtype=torch.float64, device="cuda:0"))
        B = torch.stack([b * (1 + q) for q in range(3)])
        tol = 1e-10 * float(torch.linalg.norm(b))
        xs = []
        for how in ("fp64", "mixed", "batched", "fp64"):
            x = torch.zeros_like(b)
            if how == "fp64":
                s.gmres(x, b, tol, raise_noconv=True)
            elif how == "mixed":
                s.solve_mixed(x, b, tol, raise_noconv=True)
            else:
                X = torch.zeros_like(B)
                s.solve_mixed_batched(X, B, tol, raise_noconv=True)
                x = X[0].clone()
            assert float(torch.linalg.norm(s.residual(x, b))) <= tol * (1 + 1e-9)
            xs.append(x)
            held.append(s.info()["device_bytes"])
    finally:
        s.close()
    for x in xs[1:]:
        assert float((x - xs[0]).abs().max()) <= 1e-7 * float(xs[0].abs().max())
    return held, m.nele


@pytest.mark.parametrize("mode", ["quadrature", "affine"])
def test_digits_given_back(mode, monkeypatch):
    held, nele = _run(mode, 0, monkeypatch)
    digits = nele * 16080 + 16
    for short in (1, digits // 2, digits):
        less, _ = _run(mode, held[-1] - short, monkeypatch)
        assert less[0] == held[0] and less[-1] == held[-1] - digits
    with pytest.raises(DGError, match="cudaMalloc"):
        _run(mode, held[-1] - digits - 1, monkeypatch)
