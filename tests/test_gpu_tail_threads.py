"""Two threads that rebuild contexts of different sizes side by side, as the
native request queue's workers do, and apply the FP64 V-cycle: the matrix of
its coarse tail is formed by one kernel with shared memory by the context's
size (9 KB for 125 vertices, 78 KB for 1,089), and every result is the first
one's."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from dg_nn_public_gb300 import element, mesh, sfc  # noqa: E402
from dg_nn_public_gb300.solver import DGSolver, SolverConfig  # noqa: E402


def test_contexts_of_two_sizes_in_two_threads():
    slots = []
    for kind, n in (("tet", 4), ("tri", 32)):
        m = mesh.build_mesh(kind, n, seed=4)
        s = DGSolver(m, sfc.hilbert_sfc_order(m.cg_coords), SolverConfig(), element.p3_element(m.ndim))
        s.set_build_mode("affine")
        s.build_operator()
        r = torch.tensor(np.random.default_rng(5).standard_normal(m.cg_nonods), device="cuda:0")
        slots.append((s, r, s.mg_vcycle(r).clone()))
    failed = []
    go = threading.Barrier(2)

    def work(s, r, first):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(400):
                    s.build_operator()
                    go.wait()
                    e = s.mg_vcycle(r)
                    torch.cuda.current_stream().synchronize()
                    assert torch.equal(e, first)
        except Exception as err:
            failed.append(err)
            go.abort()
    torch.cuda.synchronize()
    th = [threading.Thread(target=work, args=a) for a in slots]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not [e for e in failed if not isinstance(e, threading.BrokenBarrierError)], failed
    for s, _, _ in slots:
        s.close()
