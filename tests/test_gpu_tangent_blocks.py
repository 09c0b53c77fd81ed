"""The assembled tangent of every material form, and that it follows its state.

The blocks are compared through solves: K du = r solved on the assembled blocks
to 1e-7, K du then formed by the element product, which other tests hold against
the FP64 oracle.  FP32 products and sums leave some 1e-6 times the condition of
these systems (a few hundred): 1e-3; a wrong block leaves 1e-2 and more."""
import ctypes as C

import numpy as np
import pytest
import torch

from simul_b200 import _lib, meshgen
from simul_b200 import fem as B
from tests.golden import gen_golden as G
from tests.test_gpu_hex8 import distorted_grid

pytestmark = pytest.mark.gpu
JACOBI, TWO_LEVEL = _lib.FEM_PRECOND_JACOBI, _lib.FEM_PRECOND_TWO_LEVEL


def _j2(E):
    return B.J2Plasticity(E, 0.3, 10.0, hardening_modulus=0.02 * E)


MATS = {
    "le": lambda: B.LinearElastic(1e3, 0.3),
    "nh": lambda: B.NeoHookean(1e3, 0.3),
    "mr": lambda: B.MooneyRivlin(100.0, 30.0, 0.005),
    "fmr": lambda: B.FibreReinforcedMooneyRivlin(100.0, 30.0, 0.005, G.FIBRES, 500.0),
    "ti": lambda: B.TransverseIsotropic(1.7e3, 1.15e3, 0.3, 0.35, 330.0, fiber_direction=(1.0, 1.0, 0.0)),
    "j2": lambda: _j2(1e3),
    "mixed": lambda: {0: _j2(1e3), 1: B.MooneyRivlin(100.0, 30.0, 0.005), 2: B.LinearElastic(2e3, 0.3)},
}


class Case:
    def __init__(self, element, key, cuda, n=4):
        self.key = key
        if element == "hex8":
            self.X, conn = distorted_grid(n=n, seed=1)
        else:
            self.X, conn = meshgen.structured_tets(n, n, n, L=(float(n),) * 3)
            rng = np.random.default_rng(1)
            inner = np.all((self.X > 0.5) & (self.X < n - 0.5), axis=1)
            self.X = self.X.copy()
            self.X[inner] += 0.1 * rng.uniform(-1, 1, (int(inner.sum()), 3))
        ids = np.arange(conn.shape[0]) % 3 if key == "mixed" else None
        self.mesh = B.FEMesh(self.X.shape[0], conn.shape[0],
                             B.ElementType.HEX8 if element == "hex8" else B.ElementType.TET4, device=cuda)
        self.mesh.initialize_from_numpy(self.X, conn, material_ids=ids)
        self.fix(self.X[:, 2] == 0.0)
        self.mat = MATS[key]()
        if key == "mixed":
            B.StaticSolver(self.mesh, materials=self.mat)._bind()

    def fix(self, nodes):
        self.fixed = np.zeros(self.X.shape, dtype=bool)
        self.fixed[nodes] = True
        self.mesh.set_fixed_dofs(np.where(self.fixed.reshape(-1))[0])

    def state(self, strain, commit=False):
        """Forces at a compressed and perturbed state."""
        u = 0.005 * np.random.default_rng(3).standard_normal(self.X.shape)
        u[:, 2] -= strain * self.X[:, 2]
        u[self.fixed] = 0.0
        self.mesh.u.copy_(torch.from_numpy(u))
        if self.key == "mixed":
            self.mesh._push_bc()
            lib = _lib.load()
            B._check(lib.fem_element_forces(self.mesh.ctx, B._ptr(self.mesh.u), B._ptr(self.mesh.f), None, None),
                     self.mesh.ctx)
        else:
            self.mat.compute_nodal_forces(self.mesh)
        if commit:
            assert _lib.load().fem_commit_history(self.mesh.ctx) == 0

    def solve(self, pc=JACOBI):
        rhs = np.random.default_rng(5).standard_normal(self.X.shape)
        rhs[self.fixed] = 0.0
        r = torch.from_numpy(rhs).to(self.mesh.device)
        du = torch.zeros_like(r)
        it, rel = C.c_int32(), C.c_double()
        rc = _lib.load().fem_pcg(self.mesh.ctx, pc, B._ptr(r), B._ptr(du), 1e-7, 20000, C.byref(it), C.byref(rel))
        assert rc == 0, _lib.last_error(self.mesh.ctx)
        assert self.mesh.stats()["matvec_variant"] == "assembled"
        return du, r

    def residual(self, du, r):
        x = du.to(torch.float32)
        y = torch.empty_like(x)
        assert _lib.load().fem_tangent_matvec(self.mesh.ctx, B._ptr(x), B._ptr(y)) == 0
        return float((y.double() - r).norm() / r.norm())


@pytest.mark.parametrize("element", ["tet4", "hex8"])
@pytest.mark.parametrize("key", sorted(MATS))
def test_blocks_of_every_material(cuda, key, element):
    c = Case(element, key, cuda)
    if key in ("j2", "mixed"):
        c.state(0.02, commit=True)   # past yield (1 % strain)
    for strain in (0.03, 0.05):      # the second state reuses the tables
        c.state(strain)
        assert c.residual(*c.solve()) < 1e-3
        assert c.residual(*c.solve(TWO_LEVEL)) < 1e-3


@pytest.mark.parametrize("element", ["tet4", "hex8"])
@pytest.mark.parametrize("key", ["le", "nh"])
def test_blocks_follow_constraints_and_materials(cuda, key, element):
    """One context through a change of constraints and of materials gives the
    bits of a fresh context each time."""
    c = Case(element, key, cuda)
    other = {"le": lambda: B.LinearElastic(3e3, 0.2), "nh": lambda: B.NeoHookean(3e3, 0.2)}[key]

    def fresh(nodes, mat):
        f = Case(element, key, cuda)
        f.fix(nodes)
        f.mat = mat
        f.state(0.03)
        return f

    bottom, side = c.X[:, 2] == 0.0, c.X[:, 0] == 0.0
    for nodes, make in ((bottom, MATS[key]), (side, MATS[key]), (side, other)):
        c.fix(nodes)
        c.mat = make()
        c.state(0.03)
        f = fresh(nodes, make())
        for pc in (JACOBI, TWO_LEVEL):
            assert torch.equal(c.solve(pc)[0], f.solve(pc)[0])


def test_large_solve_matches_kernel_chain(cuda):
    """Above the sizes of the other tests: two FP32 solves to 1e-6, 1e-4,
    iterations within 5 %."""
    v = meshgen.vertebral_body(n=72, seed=1)
    rhs = np.random.default_rng(7).standard_normal(v.X.shape)
    rhs[v.fixed_mask] = 0.0
    mesh = B.FEMesh(v.n_nodes, v.n_elements, device=cuda)
    mesh.initialize_from_numpy(v.X, v.conn)
    mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
    mesh.set_coarse_options(cell=4, bf16=True, inverse="f32", max_nodes=6144)
    B.LinearElastic(1e3, 0.3).compute_nodal_forces(mesh)
    r = torch.from_numpy(rhs).to(cuda)
    out = []
    for variant in ("auto", "persistent"):
        mesh.set_matvec_variant(variant)
        du = torch.zeros_like(r)
        it, rel = C.c_int32(), C.c_double()
        rc = _lib.load().fem_pcg(mesh.ctx, TWO_LEVEL, B._ptr(r), B._ptr(du), 1e-6, 20000, C.byref(it), C.byref(rel))
        assert rc == 0, _lib.last_error(mesh.ctx)
        assert mesh.stats()["matvec_variant"] == {"auto": "assembled"}.get(variant, variant)
        out.append((du, it.value))
    (a, ia), (b, ib) = out
    assert abs(ia - ib) <= 0.05 * ib + 2
    assert float((a - b).norm() / b.norm()) < 1e-4
