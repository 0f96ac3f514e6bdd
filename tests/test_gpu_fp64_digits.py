"""FP64 products from digits on the tensor cores against the FP64 loop.

The operator is read out exactly, column by column (dg_apply of a unit vector
adds only zeros to an entry), and A x is formed in extended precision.  With
b = A x rounded to FP64, b - A x is the products' own error (and half an ulp
of b): its norm from the digit product has to be at most that of the FP64
loop (dg_residual).  Vectors: N(0, 1); smooth; magnitudes spread over 12
decades with zeros.  Meshes of 6 and 48 elements (boundary faces, one to
several warps), 1 to 64 right-hand sides (groups of 16 with remainders).

The FP64 loop is that of an affine build, whose single products stay on it;
a quadrature build's take the digits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def _operator(n, build="affine"):
    m = mesh.build_mesh("tet", n, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(3))
    s.set_kappa(np.exp(np.random.default_rng(1).standard_normal(m.nele)))
    s.set_face_kappa("harmonic")
    s.set_build_mode(build)
    s.build_operator()
    A = np.empty((s.nonods, s.nonods))
    for j in range(s.nonods):
        u = torch.zeros(s.nonods, dtype=torch.float64, device="cuda:0")
        u[j] = 1.0
        A[:, j] = s.apply(u).cpu().numpy()
    return s, A.astype(np.longdouble)


def _vectors(n, nrhs, kind):
    rng = np.random.default_rng(nrhs)
    x = rng.standard_normal((nrhs, n))
    if kind == "smooth":
        x = np.sin(np.arange(n) / n * (1 + np.arange(nrhs)[:, None]))
    elif kind == "spread":
        x = x * 10.0 ** rng.uniform(-6, 6, x.shape) * (rng.uniform(size=x.shape) > 0.2)
    return x


@pytest.mark.parametrize("n,nrhs", [(1, 64), (1, 1), (2, 17)])
def test_batched_residual_error(n, nrhs):
    s, A = _operator(n)
    for kind in ("normal", "smooth", "spread"):
        x = _vectors(s.nonods, nrhs, kind)
        b = np.stack([(A @ q.astype(np.longdouble)).astype(np.float64) for q in x])
        xt, bt = torch.tensor(x, device="cuda:0"), torch.tensor(b, device="cuda:0")
        _, res = s.solve_mixed_batched(xt.clone(), bt, 0.0, max_its=0)
        ref = np.array([float(torch.linalg.norm(s.residual(xt[q].contiguous(), bt[q].contiguous())))
                        for q in range(nrhs)])
        print(kind, nrhs, "digits / FP64 loop: max %.3f" % (res / ref).max())
        assert (res <= ref).all(), (kind, res, ref)
    s.close()


def test_batched_residual_nonfinite():
    s, _ = _operator(1)
    x = torch.randn(20, s.nonods, dtype=torch.float64, device="cuda:0")
    x[7, 3] = float("inf")
    with pytest.raises(Exception, match="non-finite"):
        s.solve_mixed_batched(x, torch.ones_like(x), 1e-10)
    s.close()


def _loop(A, x, b):
    """Norm of b - A x from an FP64 multiply-add chain per row, in column order."""
    A, r = A.astype(np.float64), np.zeros_like(b)
    cols = [np.nonzero(a)[0] for a in A]
    for i, c in enumerate(cols):
        acc = 0.0
        for j in c:
            acc += A[i, j] * x[j]
        r[i] = b[i] - acc
    return r


@pytest.mark.parametrize("n", [1, 2])
def test_single_product_flags(n):
    """dg_residual from the digits: error against extended precision at most
    the FP64 chain's, its smoothing step against the same step from that
    residual (FP64 products of 20 terms: 1e-13 of the largest), the
    preconditioner (restriction of the residual) against the affine build's
    (blocks equal to 1e-13: 1e-10 of the largest)."""
    s, A = _operator(n, "quadrature")
    a = _operator(n, "affine")[0]
    K, d = s.bdiag()
    for kind in ("normal", "smooth", "spread"):
        x = _vectors(s.nonods, 3, kind)[2]
        b = (A @ x.astype(np.longdouble)).astype(np.float64)
        xt, bt = torch.tensor(x, device="cuda:0"), torch.tensor(b, device="cuda:0")
        r = s.residual(xt, bt)
        chain = _loop(A, x, b)
        print(kind, "digits / chain: %.3f" % (float(torch.linalg.norm(r)) / np.linalg.norm(chain)))
        assert float(torch.linalg.norm(r)) <= np.linalg.norm(chain)
        y = s.apply(xt)
        assert torch.equal(y, -s.residual(xt, torch.zeros_like(xt)))
        b2 = torch.tensor(_vectors(s.nonods, 5, "normal")[4], device="cuda:0") * float(y.abs().max())
        out = torch.empty_like(xt)
        r2 = s.residual(xt, b2, x_out=out, smooth=True).view(-1, 20)
        c = torch.zeros_like(r2)
        for _ in range(3):
            c = c + (2.0 / 3.0) * (r2 - torch.bmm(K, c.unsqueeze(2)).squeeze(2)) / d
        ref = xt.view(-1, 20) + (2.0 / 3.0) * c
        assert float(torch.abs(out.view(-1, 20) - ref).max()) <= 1e-13 * float(torch.abs(ref).max())
    f = torch.tensor(_vectors(s.nonods, 3, "normal")[1], device="cuda:0")
    z, za = s.precond(f), a.precond(f)
    assert float(torch.abs(z - za).max()) <= 1e-10 * float(torch.abs(za).max())
    x = torch.zeros_like(f)
    x[5] = float("nan")
    assert not bool(torch.isfinite(s.residual(x, f)).all())
    s.close()
    a.close()
