"""FP64 products at the ends of the exponent range: x scaled by a power of two
gives the product scaled by it, bit for bit (the results stay normal numbers),
for a default build's products (digits) and an affine one's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


@pytest.mark.parametrize("build", ["quadrature", "affine"])
@pytest.mark.parametrize("kscale", [0, -400, 400])
def test_scaled_vectors(build, kscale):
    m = mesh.build_mesh("tet", 2, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(3))
    s.set_kappa(np.full(m.nele, 2.0 ** kscale))
    s.set_build_mode(build)
    s.build_operator()
    x = torch.tensor(np.random.default_rng(4).standard_normal(s.nonods), device="cuda:0")
    y = s.apply(x)
    for k in (-1000 - min(kscale, 0), -990 - min(kscale, 0), -500, 500, 900 - max(kscale, 0)):
        up = torch.tensor(np.ldexp(x.cpu().numpy(), k), device="cuda:0")
        want = np.ldexp(y.cpu().numpy(), k)
        got = s.apply(up).cpu().numpy()
        assert np.array_equal(got, want), (k, np.abs(got / want - 1).max())
        r = s.residual(up, torch.tensor(want, device="cuda:0")).cpu().numpy()
        assert np.abs(r).max() <= 2.0 ** -50 * np.abs(want).max()
    s.close()
