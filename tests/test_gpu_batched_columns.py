"""Batched solve kernels at the edges of their column groups and alignments.

Up to 32 right-hand sides compute 32 columns, more compute 64: solves with 1,
31, 32 and 33 right-hand sides reach 1e-10 ||b|| in FP64 and agree with the
single solves within 1e-7 (two approximations within the tolerance), on
meshes with remainders of the kernels' element groups, also after a solve
with the other width on the same context.

dg_smooth_scaled_batched takes cv and x_out on 8-byte boundaries: same bits
as on 16-byte ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def _solver(n):
    m = mesh.build_mesh("tet", n, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(3))
    s.build_operator()
    return s


@pytest.mark.parametrize("n,widths", [(3, (1, 33)), (5, (33, 32)), (4, (31, 64))])
def test_batched_widths(n, widths):
    s = _solver(n)
    g = torch.Generator(device="cuda:0").manual_seed(n)
    for nrhs in widths:
        f = torch.randn(nrhs, s.nonods, dtype=torch.float64, device="cuda:0", generator=g)
        b = torch.stack([s.rhs(q.contiguous()) for q in f])
        tol = 1e-10 * torch.linalg.norm(b, dim=1).cpu().numpy()
        x = torch.zeros_like(b)
        _, res = s.solve_mixed_batched(x, b, tol, raise_noconv=True)
        assert (res <= tol).all()
        for q in sorted({0, nrhs - 1}):
            r = s.residual(x[q].contiguous(), b[q].contiguous())
            assert float(torch.linalg.norm(r)) <= tol[q] * (1 + 1e-9)
            x1 = torch.zeros_like(b[q])
            s.solve_mixed(x1, b[q].contiguous(), float(tol[q]))
            assert float(torch.abs(x[q] - x1).max() / torch.abs(x1).max()) < 1e-7
    s.close()


def test_scaled_step_alignment():
    s = _solver(3)
    n = s.nonods * 64
    g = torch.Generator(device="cuda:0").manual_seed(1)
    x = torch.randn(n, device="cuda:0", generator=g)
    cv = torch.randn(n, device="cuda:0", generator=g)
    out = s.smooth_scaled_batched(x, cv)
    pad_c, pad_o = torch.empty(n + 2, device="cuda:0"), torch.empty(n + 2, device="cuda:0")
    pad_c[2:].copy_(cv)
    s.smooth_scaled_batched(x, pad_c[2:], pad_o[2:])
    assert torch.equal(pad_o[2:], out)
    s.close()
