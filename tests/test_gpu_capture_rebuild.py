"""Single stages captured by the caller into a CUDA graph: a replay after a
rebuild of the operator gives the rebuilt operator's result, and a first call
under capture leaves later direct calls right.  The FP64 product and the
V-cycle keep data formed per build (digits of the blocks, the matrix of the
coarse tail), which a captured call cannot refresh.  dg_apply against the
direct call: two summation orders of 100 terms, 1e-13 of the largest; the
V-cycle: the parity tests' 1e-12."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402

DEV = "cuda:0"


def _solver(kind, n):
    m = mesh.build_mesh(kind, n, seed=4)
    s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(pre_smooth_its=2, post_smooth_its=2),
                 element.p3_element(m.ndim))
    s.build_operator()
    return m, s


def _rebuild(m, s, seed, mode):
    s.set_kappa(np.exp(np.random.default_rng(seed).standard_normal(m.nele)))
    s.set_face_kappa("harmonic")
    s.set_build_mode(mode)
    s.build_operator()


def _close(a, b, tol):
    assert float((a - b).abs().max()) <= tol * float(b.abs().max())


@pytest.mark.parametrize("mode", ["quadrature", "affine"])
def test_apply(mode):
    m, s = _solver("tet", 3)
    x = torch.tensor(np.random.default_rng(1).standard_normal(s.nonods), device=DEV)
    y = torch.zeros_like(x)
    s.apply(x, y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s.apply(x, y)
    for seed in (2, 3):
        _rebuild(m, s, seed, mode)
        g.replay()
        torch.cuda.synchronize()
        _close(y, s.apply(x), 1e-13)
    s.close()


@pytest.mark.parametrize("warm", [True, False])
@pytest.mark.parametrize("kind,n,rows", [("tri", 9, ""), ("tet", 4, ""), ("tet", 8, ""), ("tet", 8, "100"), ("tet", 1, "")])
def test_vcycle(kind, n, rows, warm, monkeypatch):
    if rows:
        monkeypatch.setenv("DG_TAIL_MAX64", rows)
    m, s = _solver(kind, n)
    r = torch.tensor(np.random.default_rng(1).standard_normal(m.cg_nonods), device=DEV)
    e = torch.zeros_like(r)
    if warm:
        s.mg_vcycle(r)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        e.copy_(s.mg_vcycle(r))
    direct = s.mg_vcycle(r).clone()
    g.replay()
    torch.cuda.synchronize()
    _close(direct, e, 1e-12)
    for seed in (2, 3):
        _rebuild(m, s, seed, "affine")
        g.replay()
        torch.cuda.synchronize()
        got = e.clone()
        _close(got, s.mg_vcycle(r), 1e-12)
    s.close()
