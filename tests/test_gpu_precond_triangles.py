"""Precision of the mixed preconditioner's block copies on triangles: FP32
with the default options (tetrahedra keep BF16).

One smoothing step x + w A_ee^-1 (b - A x) through dg_smooth_pc against the
same step from the FP64 blocks, with the tolerance of the tetrahedra's FP32 step:
1e-5 of max |x_out| (2^-24 per operation, 40 + 10 terms a row, element blocks
with condition numbers below 1e3 damped by their own inverse); BF16 blocks
give ~1e-2.  Sizes: below one element group of 16, a remainder, many groups."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("n", [2, 5, 16])
def test_triangle_smoothing_is_fp32(n):
    m = mesh.build_mesh("tri", n, seed=3)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(2))
    s.build_operator()
    g = torch.Generator(device="cuda:0").manual_seed(3)
    x = torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g)
    b = torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g)
    K, _ = s.bdiag()
    r = s.residual(x, b).view(m.nele, m.nloc, 1)
    ref = x + 0.8 * torch.linalg.solve(K, r).view(-1)
    out = s.smooth_pc(x.float().contiguous(), b.float().contiguous())
    assert float(torch.abs(out.double() - ref).max() / torch.abs(ref).max()) < 1e-5
    s.close()
