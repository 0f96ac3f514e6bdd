"""FP64 products where the diffusivity jumps: b - A x of the single product (a
default build's dg_residual, from digits) and of the batched one, with x the
solution of the jump problem and b = A x rounded to FP64, so that what is left
is the products' own error.

The operator's rows are read out by unit vectors (exact, checked against the
block diagonal), A x is formed in extended precision.  Bound of every row:
16 x 2^-53 sum |a||x|, where an FP64 chain of 100 terms may be off by 100 and
measures 4 to 12; and half an ulp of b.  Meshes of 162 elements; contrasts up
to 1e10, harmonic and arithmetic face means, spread and localised vectors."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300._capi import DGError  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402

DEV = "cuda:0"


def _solver(n, contrast, mean="harmonic"):
    m = mesh.build_mesh("tet", n, seed=2)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(3))
    s.set_kappa(np.where(m.x_ref_in[:, 0, :4].mean(1) < 0.5, 1.0, 1.0 / contrast))
    s.set_face_kappa(mean)
    s.build_operator()
    return m, s


def _rows(m, s):
    """Rows of A as (nele, 20, 100) over the element and its neighbours, and
    those elements (nele, 5), -1 at the boundary."""
    nb = np.asarray(m.nbf).reshape(m.nele, 4)
    nb = np.concatenate([np.arange(m.nele)[:, None], np.where(nb >= 0, nb // 4, -1)], 1)
    rows = np.zeros((m.nele, 20, 5, 20))
    u = torch.zeros(s.nonods, dtype=torch.float64, device=DEV)
    for j in range(s.nonods):
        u[j] = 1.0
        y = s.apply(u).cpu().numpy().reshape(m.nele, 20)
        u[j] = 0.0
        for b, e in zip(*np.nonzero((nb == j // 20).T)):
            rows[e, :, b, j % 20] = y[e]
    return rows.reshape(m.nele, 20, 100), nb


def _gather(x, nb):
    X = x.reshape(-1, 20)[np.maximum(nb, 0)]
    X[nb < 0] = 0.0
    return X.reshape(len(nb), 100)


def _vectors(m, s, rows, nb):
    A = np.zeros((s.nonods, s.nonods))
    for e in range(m.nele):
        for b in range(5):
            if nb[e, b] >= 0:
                A[20 * e:20 * e + 20, 20 * nb[e, b]:20 * nb[e, b] + 20] = rows[e][:, 20 * b:20 * b + 20]
    f = s.rhs(torch.ones(s.nonods, dtype=torch.float64, device=DEV)).cpu().numpy()
    rng = np.random.default_rng(3)
    near = np.zeros(s.nonods)
    near[20 * (m.nele // 2):20 * (m.nele // 2) + 40] = rng.standard_normal(40)
    return {"solution": np.linalg.solve(A, f), "normal": rng.standard_normal(s.nonods), "local": near,
            "spread": rng.standard_normal(s.nonods) * 10.0 ** rng.uniform(-6, 6, s.nonods)}


@pytest.mark.parametrize("contrast,mean", [(1.0, "harmonic"), (1e2, "harmonic"), (1e4, "harmonic"), (1e6, "harmonic"),
                                           (1e8, "harmonic"), (1e10, "harmonic"), (30.0, "mean"),
                                           (1e6, "mean")])
def test_rows_as_exact_as_the_loop(contrast, mean):
    m, s = _solver(3, contrast, mean)
    rows, nb = _rows(m, s)
    K, _ = s.bdiag()
    assert np.array_equal(rows[:, :, :20], K.cpu().numpy())
    L = rows.astype(np.longdouble)
    vec = _vectors(m, s, rows, nb)
    for k, x in vec.items():
        X = _gather(x, nb)
        ax = np.einsum("emj,ej->em", L, X.astype(np.longdouble))
        b = ax.astype(np.float64)
        bound = 2.0 ** -53 * (16 * np.einsum("emj,ej->em", np.abs(rows), np.abs(X)) + np.abs(b))
        xt, bt = torch.tensor(x, device=DEV), torch.tensor(b.reshape(-1), device=DEV)
        r = s.residual(xt, bt).cpu().numpy().reshape(m.nele, 20)
        over = (np.abs(r) / np.maximum(bound, 1e-300)).max()
        print("%g %s %s: row error / bound %.3f" % (contrast, mean, k, over))
        assert over <= 1.0, (k, over)
    # the batched product, all vectors together and 17 of one kind: its norms
    for xs in (np.stack(list(vec.values())), np.stack([vec["solution"] * (1 + q) for q in range(17)])):
        bs, bounds = [], []
        for x in xs:
            X = _gather(x, nb)
            bs.append(np.einsum("emj,ej->em", L, X.astype(np.longdouble)).astype(np.float64).reshape(-1))
            bounds.append(np.linalg.norm(2.0 ** -53 * (16 * np.einsum("emj,ej->em", np.abs(rows), np.abs(X)) +
                                                       np.abs(bs[-1].reshape(-1, 20)))))
        xt, bt = torch.tensor(xs, device=DEV), torch.tensor(np.stack(bs), device=DEV)
        try:
            _, res = s.solve_mixed_batched(xt, bt, 0.0, max_its=0)
        except Exception as err:   # no mixed preconditioner for this operator
            assert mean == "mean" and "pivot" in str(err)
            break
        print("batched", res / np.array(bounds))
        assert (res <= np.array(bounds)).all()
    s.close()


def test_batched_rows_far_from_a_large_value():
    """Each right-hand side has one value of 2^40 in one element, zeros in the
    two rings around it and N(0, 1) beyond: the rows that see the large value
    are exact, so the norm is the other rows' error."""
    m, s = _solver(3, 1.0)
    rows, nb = _rows(m, s)
    L = rows.astype(np.longdouble)
    rng = np.random.default_rng(5)
    xs, bs, bounds = [], [], []
    for q in range(20):
        ring = {8 * q}
        for _ in range(2):
            ring |= {int(k) for e in ring for k in nb[e] if k >= 0}
        x = rng.standard_normal((m.nele, 20))
        x[sorted(ring)] = 0.0
        x[8 * q, q] = 2.0 ** 40
        X = _gather(x, nb)
        b = np.einsum("emj,ej->em", L, X.astype(np.longdouble)).astype(np.float64)
        bound = 2.0 ** -53 * (16 * np.einsum("emj,ej->em", np.abs(rows), np.abs(X)) + np.abs(b))
        bounds.append(np.linalg.norm(bound[np.abs(X).max(1) < 1e3]))
        xs.append(x.reshape(-1))
        bs.append(b.reshape(-1))
    _, res = s.solve_mixed_batched(torch.tensor(np.stack(xs), device=DEV), torch.tensor(np.stack(bs), device=DEV), 0.0,
                                   max_its=0)
    print(res / np.array(bounds))
    assert (res <= np.array(bounds)).all()
    s.close()


@pytest.mark.parametrize("contrast", [1e6, 1e8])
def test_solves_meet_the_tolerance(contrast):
    """Mixed, FP64 and batched solves to 1e-10, the residual taken by the FP64
    loop (an affine build's dg_residual)."""
    m, s = _solver(4, contrast)
    _, a = _solver(4, contrast)
    a.set_build_mode("affine")
    a.build_operator()
    b = s.rhs(torch.ones(s.nonods, dtype=torch.float64, device=DEV))
    bn = float(torch.linalg.norm(b))
    for how in ("mixed", "batched", "fp64"):
        x = torch.zeros_like(b)
        if how == "mixed":
            s.solve_mixed(x, b, 1e-10 * bn, max_its=2000, raise_noconv=True)
        elif how == "fp64":
            s.gmres(x, b, 1e-10 * bn, max_its=6000, raise_noconv=True)
        else:
            X = torch.zeros(2, s.nonods, dtype=torch.float64, device=DEV)
            B = torch.stack([b, 2.0 * b])
            s.solve_mixed_batched(X, B, 1e-10 * torch.linalg.norm(B, dim=1).cpu().numpy(), raise_noconv=True)
            x = X[0].contiguous()
        res = float(torch.linalg.norm(a.residual(x, b))) / bn
        print("%s at %g: %.3e" % (how, contrast, res))
        assert res <= 1.01e-10
    s.close()
    a.close()
