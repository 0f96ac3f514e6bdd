"""Kernels that prepare the mixed preconditioner after an operator build: the
one-pass reduced-precision copies (four elements per CTA) and the blocked
inverse of the dense coarse level (steps of 32 rows, tiles of 64).

Copies: one smoothing step through dg_smooth_pc (scaled faces) against the
FP64 blocks, tolerance 3e-2 of max |x_out| as for the other BF16 steps, and
the FP32 apply against the FP64 one, 1e-6 of max |y| (100 products, 2^-24
each).  Meshes of 6, 48 and 162 elements: remainders 2, 0 and 2 of four.

Inverse: the FP32 preconditioner with the blocked inverse against the
one-pivot FP64 form, 1e-4 of its max entry, with 4 to 81 rows: below one
step, a remainder, whole steps, two tiles."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def _solver(kind, n):
    m = mesh.build_mesh(kind, n, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.build_operator()
    return m, s


@pytest.mark.parametrize("n", [1, 2, 3])
def test_one_pass_copies(n):
    m, s = _solver("tet", n)
    g = torch.Generator(device="cuda:0").manual_seed(3)
    x = torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g)
    b = torch.randn(s.nonods, dtype=torch.float64, device="cuda:0", generator=g)
    K, _ = s.bdiag()
    ref = x + 0.8 * torch.linalg.solve(K, s.residual(x, b).view(m.nele, m.nloc, 1)).view(-1)
    out = s.smooth_pc(x.float().contiguous(), b.float().contiguous())
    assert float(torch.abs(out.double() - ref).max() / torch.abs(ref).max()) < 3e-2
    y = s.apply(x.float().double().contiguous())
    y32 = s.apply_f32(x.float().contiguous())
    assert float(torch.abs(y32.double() - y).max() / torch.abs(y).max()) < 1e-6
    s.close()


@pytest.mark.parametrize("kind,n", [("tri", 1), ("tri", 4), ("tet", 2), ("tri", 7), ("tet", 3), ("tri", 8)])
def test_blocked_inverse_sizes(kind, n, monkeypatch):
    out = {}
    for fp64 in ("0", "1"):
        monkeypatch.setenv("DG_DENSE_FP64", fp64)
        _, s = _solver(kind, n)
        g = torch.Generator(device="cuda:0").manual_seed(3)
        out[fp64] = s.precond_f32(torch.randn(s.nonods, dtype=torch.float32, device="cuda:0", generator=g)).clone()
        s.close()
    assert float(torch.abs(out["0"] - out["1"]).max() / torch.abs(out["1"]).max()) < 1e-4
