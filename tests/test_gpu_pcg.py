"""The persistent PCG kernel on the assembled tangent (fem_pcg.cu, fem_asm.cu).

Small systems against the FP64 oracle's direct solve, as the kernel chain's
tests do (FP32 vectors, residual to 1e-7: 1e-5); larger ones, where the matrix
or the coarse inverse no longer stays in shared memory, against the kernel
chain (two FP32 solves to 1e-6: 1e-4, iterations within 5 %).
"""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import fem_oracle as O
from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu
PC = {"jacobi": _lib.FEM_PRECOND_JACOBI, "two_level": _lib.FEM_PRECOND_TWO_LEVEL}


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _mesh(X, conn, fixed, cuda, E=1e3):
    mesh = B.FEMesh(X.shape[0], conn.shape[0], device=cuda)
    mesh.initialize_from_numpy(X, conn)
    mesh.set_fixed_dofs(np.where(fixed.reshape(-1))[0])
    mat = B.LinearElastic(E, 0.3)
    mat.compute_nodal_forces(mesh)
    return mesh


def _solve(mesh, pc, rhs, rtol, max_iterations=20000):
    r = torch.from_numpy(rhs).to(mesh.device)
    du = torch.zeros_like(r)
    it, rel = C.c_int32(), C.c_double()
    rc = _lib.load().fem_pcg(mesh.ctx, PC[pc], B._ptr(r), B._ptr(du), rtol, max_iterations, C.byref(it), C.byref(rel))
    return rc, du.cpu().numpy(), it.value, rel.value


def _rhs(fixed, seed):
    rhs = np.random.default_rng(seed).standard_normal(fixed.shape)
    rhs[fixed] = 0.0
    return rhs


def _oracle(X, conn, fixed, rhs):
    m = O.Mesh(X, conn)
    F = O.deformation_gradient(np.zeros_like(X), conn.astype(np.int64), m.dNdX)
    return O.solve_tangent(O.Material("linear_elastic", E=1e3, nu=0.3), F, None, m, rhs, fixed)


# grids around the edges of a slice (32 rows) and of a CTA (64 rows)
@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 2, 2), (3, 3, 3), (6, 2, 2), (15, 1, 1), (7, 3, 2)])
def test_jacobi_small_grids_match_oracle(cuda, grid):
    X, conn = meshgen.structured_tets(*grid, L=(float(grid[0]), float(grid[1]), float(grid[2])))
    fixed = np.zeros(X.shape, dtype=bool)
    fixed[X[:, 0] == 0.0] = True
    fixed[np.argmax(X.sum(1)), 1] = True   # one DOF of a node
    rhs = _rhs(fixed, 3)
    mesh = _mesh(X, conn, fixed, cuda)
    rc, u, it, rel = _solve(mesh, "jacobi", rhs, 1e-7)
    assert rc == 0 and rel <= 1e-7, _lib.last_error(mesh.ctx)
    assert mesh.stats()["matvec_variant"] == "assembled"
    assert np.all(u[fixed] == 0.0)
    assert _rel(u, _oracle(X, conn, fixed, rhs)) < 1e-5
    rc2, u2, it2, _ = _solve(mesh, "jacobi", rhs, 1e-7)
    assert rc2 == 0 and it2 == it and np.array_equal(u, u2)   # bitwise repeatable


# cell 4: full coarse rows; cell 1: 3,030 coarse DOFs, packed tiles
@pytest.mark.parametrize("cell", [1, 4])
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("block", [False, True])
def test_two_level_matches_oracle(cuda, cell, bf16, block):
    v = meshgen.vertebral_body(n=12)
    rhs = _rhs(v.fixed_mask, 5)
    mesh = _mesh(v.X, v.conn, v.fixed_mask, cuda)
    mesh.set_coarse_options(cell=cell, bf16=bf16)
    mesh.set_block_smoother(block)
    rc, u, it, rel = _solve(mesh, "two_level", rhs, 1e-7)
    assert rc == 0 and rel <= 1e-7, _lib.last_error(mesh.ctx)
    assert mesh.stats()["matvec_variant"] == "assembled" and mesh.coarse_info()["jacobi_fallbacks"] == 0
    assert _rel(u, _oracle(v.X, v.conn, v.fixed_mask, rhs)) < 1e-5
    rc2, u2, it2, _ = _solve(mesh, "two_level", rhs, 1e-7)
    assert rc2 == 0 and it2 == it and np.array_equal(u, u2)


# 40: matrix in shared memory, 52: part of it, 64: streamed with the tiles; FP32 tiles at 40
@pytest.mark.parametrize("n,cell,bf16", [(40, 8, False), (40, 3, False), (52, 8, False), (64, 4, True)])
def test_large_solves_match_kernel_chain(cuda, n, cell, bf16):
    v = meshgen.vertebral_body(n=n, seed=1)
    rhs = _rhs(v.fixed_mask, 7)
    out = []
    for chain in (False, True):
        mesh = _mesh(v.X, v.conn, v.fixed_mask, cuda)
        mesh.set_coarse_options(cell=cell, bf16=bf16, inverse="f32", max_nodes=6144)
        if chain:
            mesh.set_whole_solve_graph(False)
        rc, u, it, _ = _solve(mesh, "two_level", rhs, 1e-6)
        assert rc == 0, _lib.last_error(mesh.ctx)
        assert (mesh.stats()["matvec_variant"] == "assembled") == (not chain)
        out.append((u, it))
    assert abs(out[0][1] - out[1][1]) <= max(2, 0.05 * out[1][1])
    assert _rel(out[0][0], out[1][0]) < 1e-4


def test_end_states(cuda):
    """Iteration limit, zero right-hand side, non-finite right-hand side and a
    node without elements end as in the kernel chain."""
    X, conn = meshgen.structured_tets(4, 3, 3)
    X = np.concatenate([X, [[9.0, 9.0, 9.0]]])   # no element on the last node
    fixed = np.zeros(X.shape, dtype=bool)
    fixed[X[:, 0] == 0.0] = True
    rhs = _rhs(fixed, 9)
    rhs[-1] = 0.0
    for pc in ("jacobi", "two_level"):
        mesh = _mesh(X, conn, fixed, cuda)
        rc, u, it, _ = _solve(mesh, pc, rhs, 1e-7, 3)
        assert rc == _lib.FEM_NOT_CONVERGED and it == 3
        rc, u, it, _ = _solve(mesh, pc, np.zeros_like(rhs), 1e-7)
        assert rc == 0 and it == 0 and np.all(u == 0.0)
        bad = rhs.copy()
        bad[np.argmin(fixed[:, 0]), 0] = np.inf
        rc, _, it, _ = _solve(mesh, pc, bad, 1e-7)
        assert rc == _lib.FEM_ERR_NAN and it == 0
        rc, u, _, rel = _solve(mesh, pc, rhs, 1e-7)
        assert rc == 0 and rel <= 1e-7
        # the coarse correction moves a node without stiffness along (as in the chain), Jacobi leaves it
        assert pc == "two_level" or np.all(u[-1] == 0.0)
