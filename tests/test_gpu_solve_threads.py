"""Solves of several contexts from threads of their own on one GPU: the
displacements of the same solves one after another, and with more than two at
once their kernel chains overlap instead of one persistent kernel after another."""
import threading

import numpy as np
import pytest
import torch

from simul_b200 import meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu


class Body:
    def __init__(self, seed, cuda, element):
        v = meshgen.vertebral_body(n=20, seed=seed, element=element)
        with torch.cuda.stream(torch.cuda.Stream()):
            self.mesh = B.FEMesh(v.n_nodes, v.n_elements,
                                 B.ElementType.HEX8 if element == "hex8" else B.ElementType.TET4, device=cuda)
            self.mesh.initialize_from_numpy(v.X, v.conn)
            idx = np.where(v.fixed_mask.reshape(-1))[0]
            self.mesh.set_fixed_dofs(idx, (0.3 * v.fixed_vals).reshape(-1)[idx])
            self.mat = B.J2Plasticity(v.E, 0.3, 100.0, hardening_modulus=0.02 * v.E)
            self.solver = B.StaticSolver(self.mesh, self.mat, tol=1e-9)
            torch.cuda.synchronize()

    def solve(self):
        with torch.cuda.stream(torch.cuda.Stream()):
            self.mesh.u.zero_()
            self.mat.reset_state()
            torch.cuda.current_stream().synchronize()
            res = self.solver.solve(verbose=False)
            return bool(res["converged"]), self.mesh.u.clone().cpu()


@pytest.mark.parametrize("element", ["tet4", "hex8"])
@pytest.mark.parametrize("k", [2, 4])
def test_contexts_in_threads(cuda, k, element):
    bodies = [Body(i, cuda, element) for i in range(k)]
    want = [b.solve() for b in bodies]
    assert all(ok for ok, _ in want)
    assert all(b.mesh.stats()["matvec_variant"] == "assembled" for b in bodies)
    got = [None] * k
    together = threading.Barrier(k)

    def work(i):
        for _ in range(6):
            together.wait(60)
            got[i] = bodies[i].solve()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(k)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    for (ok, u), (_, u0) in zip(got, want):
        # solves to a residual of 1e-9, sums associated differently
        assert ok and float((u - u0).norm() / u0.norm()) < 1e-7
    chains = sum(b.mesh.stats()["whole_solve_graphs"] for b in bodies)
    assert chains == 0 if k == 2 else chains > 0
