"""HEX8 solves on the assembled tangent (persistent PCG): the blocks of the 28
vertex pairs of distorted elements for every material form, against the FP64
oracle's direct solve (FP32 vectors, residual to 1e-7: 1e-5 by the condition
of these small systems), and larger bodies against the kernel chain on element
products (two FP32 solves to 1e-6: 1e-4, iterations within 5 %)."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import fem_oracle as O
from simul_b200 import _lib, meshgen
from simul_b200 import fem as B
from tests.test_gpu_hex8 import MATS, distorted_grid, hex_mesh

pytestmark = pytest.mark.gpu


def _solve(mesh, pc, rhs, rtol):
    r = torch.from_numpy(rhs).to(mesh.device)
    du = torch.zeros_like(r)
    it, rel = C.c_int32(), C.c_double()
    rc = _lib.load().fem_pcg(mesh.ctx, pc, B._ptr(r), B._ptr(du), rtol, 20000, C.byref(it), C.byref(rel))
    assert rc == 0, _lib.last_error(mesh.ctx)
    return du.cpu().numpy(), it.value


@pytest.mark.parametrize("key", ["nh", "mr", "fmr", "le", "ti"])
@pytest.mark.parametrize("n", [1, 2, 5])
def test_assembled_hex_solve_matches_oracle(cuda, key, n):
    X, conn = distorted_grid(n=n, seed=n)
    fixed = np.zeros(X.shape, dtype=bool)
    fixed[X[:, 0] == 0.0] = True
    fixed[X[:, 0] == float(n), 1] = True          # one direction only
    rng = np.random.default_rng(n)
    u = 0.01 * rng.standard_normal(X.shape)
    u[fixed] = 0.0
    rhs = rng.standard_normal(X.shape)
    rhs[fixed] = 0.0
    mesh = hex_mesh(X, conn, cuda)
    mesh.set_fixed_dofs(np.where(fixed.reshape(-1))[0])
    mesh.u.copy_(torch.from_numpy(u))
    gpu_mat, om = MATS[key][0](), MATS[key][1]()
    gpu_mat.compute_nodal_forces(mesh)
    du, _ = _solve(mesh, _lib.FEM_PRECOND_JACOBI, rhs, 1e-7)
    assert mesh.stats()["matvec_variant"] == "assembled"
    m = O.Mesh(X, conn)
    F = O.deformation_gradient(u, m.qconn, m.dNdX)
    want = O.solve_tangent(om, F, None, m, rhs, fixed)
    assert np.linalg.norm(du - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("n,cell,bf16", [(16, 4, False), (33, 4, True), (40, 8, False)])
def test_assembled_hex_solve_matches_kernel_chain(cuda, n, cell, bf16):
    v = meshgen.vertebral_body(n=n, seed=2, element="hex8")
    rhs = np.random.default_rng(n).standard_normal(v.fixed_mask.shape)
    rhs[v.fixed_mask] = 0.0
    out = []
    for chain in (False, True):
        mesh = hex_mesh(v.X, v.conn, cuda)
        mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
        mesh.set_coarse_options(cell=cell, bf16=bf16)
        if chain:
            mesh.set_programmatic_launch(True)
        mat = B.J2Plasticity(v.E, 0.3, 100.0, hardening_modulus=0.02 * v.E)
        mat.compute_nodal_forces(mesh)
        out.append(_solve(mesh, _lib.FEM_PRECOND_TWO_LEVEL, rhs, 1e-6))
        assert (mesh.stats()["matvec_variant"] == "assembled") == (not chain)
    (a, ia), (b, ib) = out
    assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)
    assert abs(ia - ib) <= 0.05 * ib + 2
