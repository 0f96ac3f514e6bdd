"""The right-hand side kernels against the quadrature in NumPy: the mass
product where the element map is straight (sizes at and around the 16 or 32
elements of a block), nearly straight (the FP32 correction), curved, or the
source out of FP32's range (two FP64 passes), and Dirichlet and Neumann faces
in one launch with elements that have up to three of them.

Both sides round sums of at most 2 N VG = 960 products in an order of their
own, on geometry that is itself rounded (coordinates of order 1, elements of
1 / n): 1e-12 of the largest entry."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.element import drst_duv  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def _reference(m, el, eta, f, g, gn):
    D, N = m.ndim, m.nloc
    X = np.asarray(m.x_ref_in)                                     # (e, a, n)
    J = np.einsum("ing,ean->egia", el.nlx.reshape(D, N, -1), X)
    detw = np.linalg.det(J) * el.weight
    b = np.einsum("mg,eg,ng,en->em", el.n, detw, el.n, f.reshape(-1, N), optimize=True)
    dr = drst_duv(D).reshape(D + 1, D, D - 1)
    sn = el.sn.reshape(D + 1, N, -1)
    snlx = el.snlx.reshape(D + 1, D, N, -1)
    for k in np.flatnonzero(np.isin(m.glb_bcface_type, (0, 1))):
        e, q = divmod(int(k), D + 1)
        Jf = np.einsum("ing,an->gia", snlx[q], X[e])
        T = np.einsum("ic,gia->gca", dr[q], Jf)
        n = np.cross(T[:, 0], T[:, 1]) if D == 3 else np.stack([T[:, 0, 1], -T[:, 0, 0]], 1)
        sdet = np.linalg.norm(n, axis=1)
        n /= sdet[:, None]
        out = np.einsum("ng,an->ga", sn[q], X[e]).mean(0) - X[e].mean(1)
        n *= np.sign(n @ out)[:, None]
        w = sdet * el.sweight
        data = (g if m.glb_bcface_type[k] == 0 else gn)
        if data is None:
            continue
        dq = w * (data.reshape(-1, N)[e] @ sn[q])
        if m.glb_bcface_type[k] == 1:
            b[e] += sn[q] @ dq
        else:
            h = np.sqrt(w.sum()) if D == 3 else w.sum()
            grad = np.einsum("gai,ing->gan", np.linalg.inv(Jf), snlx[q])
            b[e] += np.einsum("gn,g->n", eta / h * sn[q].T - np.einsum("gan,ga->gn", grad, n), dq)
    return b.reshape(-1)


@pytest.mark.parametrize("kind,n", [("tet", 1), ("tet", 2), ("tet", 3), ("tri", 1), ("tri", 4), ("tri", 9)])
@pytest.mark.parametrize("curve", [0.0, 1e-11, 1e-3])
@pytest.mark.parametrize("source", [1.0, 1e-25])
def test_rhs(kind, n, curve, source):
    m = mesh.build_mesh(kind, n, seed=2)
    m.x_ref_in = np.ascontiguousarray(m.x_ref_in + curve * np.sin(3.0 * m.x_ref_in[:, ::-1]))
    bnd = np.flatnonzero(m.glb_bcface_type == 0)
    m.glb_bcface_type[bnd[::3]] = 1
    el = element.p3_element(m.ndim)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(), el)
    s.build_operator()
    rng = np.random.default_rng(n)
    f, g, gn = (v * rng.standard_normal(s.nonods) for v in (source, 1.0, 1.0))
    dev = [torch.tensor(v, device="cuda:0") for v in (f, g, gn)]
    for use_g, use_gn in ((0, 0), (1, 0), (0, 1), (1, 1)):
        ref = _reference(m, el, s.cfg.eta_e, f, g if use_g else None, gn if use_gn else None)
        out = s.rhs(dev[0], dev[1] if use_g else None, dev[2] if use_gn else None).cpu().numpy()
        assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()
    s.close()
