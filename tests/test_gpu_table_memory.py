"""The assembled tangent's tables are optional: where the device memory does not
hold them a solve runs as the kernel chain, keeps nothing of a half-built set,
and a later solve does not try again; where a required buffer finds no room,
they make it."""
import types

import numpy as np
import pytest
import torch

from simul_b200 import batch, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu


class Body:
    def __init__(self, n, element, cuda, **coarse):
        v = meshgen.vertebral_body(n=n, element=element)
        self.mesh = B.FEMesh(v.n_nodes, v.n_elements,
                             B.ElementType.HEX8 if element == "hex8" else B.ElementType.TET4, device=cuda)
        self.mesh.initialize_from_numpy(v.X, v.conn)
        idx = np.where(v.fixed_mask.reshape(-1))[0]
        self.mesh.set_fixed_dofs(idx, (0.2 * v.fixed_vals).reshape(-1)[idx])
        self.mesh.set_coarse_options(**coarse)
        self.mat = B.LinearElastic(v.E, 0.3)
        self.mat.compute_nodal_forces(self.mesh)
        self.solver = B.StaticSolver(self.mesh, self.mat, tol=1e-9)

    def solve(self):
        self.mesh.u.zero_()
        assert self.solver.solve(verbose=False)["converged"]
        return self.mesh.u.clone()

    def bytes(self):
        return self.mesh.info()["device_bytes"]


def _chain(*bodies):
    """All bodies as kernel chains (a batch of several workers): what the chain
    needs is allocated then, the tables are not."""
    for b in bodies:
        b.mesh.u.zero_()
        B._check(B._lib.load().fem_set_displacement(b.mesh.ctx, B._ptr(b.mesh.u)))
    out = batch.solve_batch([types.SimpleNamespace(mesh=b.mesh, ctx=b.mesh.ctx) for b in bodies], load_steps=1,
                            tol=1e-9)
    assert all(o["converged"] for o in out["instances"])
    return [b.mesh.u.clone() for b in bodies]


def _fill(left):
    """Takes device memory until about ``left`` bytes are free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    for step in (1 << 30, 2 << 20):
        n = (torch.cuda.mem_get_info()[0] - left) // step
        if n > 0:
            held.append(torch.empty(n * step, dtype=torch.uint8, device="cuda"))
    return held


def _close(a, b):
    # two solves to a residual of 1e-9, products and sums associated differently
    return float((a - b).norm() / b.norm()) < 1e-7


@pytest.mark.parametrize("n,element", [(56, "tet4"), (48, "hex8")])
def test_solve_without_room_for_the_tables(cuda, n, element):
    body, other = Body(n, element, cuda), Body(12, element, cuda)
    want = _chain(body, other)[0]
    before = body.bytes()
    held = _fill(24 << 20)   # the blocks alone take 38 MB and more
    try:
        got = [body.solve() for _ in range(2)]
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert body.mesh.stats()["matvec_variant"] != "assembled"
    assert body.bytes() == before
    assert all(_close(u, want) for u in got)


def test_required_buffers_take_the_room_of_the_tables(cuda):
    """A new lattice that fits only where the tables go."""
    body, other = Body(56, "tet4", cuda), Body(12, "tet4", cuda)
    twin = Body(56, "tet4", cuda, cell=6)
    _chain(body, other)
    want = _chain(twin, other)[0]
    without = body.bytes()
    body.solve()
    assert body.mesh.stats()["matvec_variant"] == "assembled"
    tables = body.bytes() - without
    body.mesh.set_coarse_options(cell=6)     # drops the lattice and its buffers
    nd = -(-twin.mesh.coarse_info()["coarse_dofs"] // 64) * 64
    need = 16 * nd * nd                      # the inversion's work space, beside the lattice's own buffers
    need += twin.bytes() - (body.bytes() - tables)
    assert tables > 32 << 20
    held = _fill(need + (16 << 20) - tables // 2)
    try:
        got = body.solve()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert body.mesh.stats()["matvec_variant"] != "assembled"
    assert _close(got, want)
