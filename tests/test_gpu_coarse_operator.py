"""The two-level preconditioner against its definition in 64 bits.

The first CG iterate of a zero start is alpha z with z = S r + P Ac^-1 P^T r:
the lattice's trilinear interpolation P, Ac = P^T K P over free DOFs (a unit
diagonal where none reaches), the smoother S and alpha = r.z / z.K z, all formed
here by scipy from the oracle's stiffness.  Bodies whose lattice cells hold a few
to some thousand elements: remainders of a chunk of 32, several chunks and
slices.  FP32 blocks and inverses leave 1e-7 times the condition of Ac (450 here,
26,000 on the finest lattice, of which a random r excites little): 1e-3.  One
element missing from Ac changes z by 1.5e-3 and more."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch
from scipy.sparse.linalg import spsolve

from oracle import fem_oracle as O
from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu
N = 12


@pytest.fixture(scope="module", params=["tet4", "hex8"])
def body(request):
    v = meshgen.vertebral_body(n=N, seed=3, element=request.param)
    m = O.Mesh(v.X, v.conn)
    conn = np.asarray(m.qconn, dtype=np.int64)
    F = O.deformation_gradient(np.zeros_like(v.X), conn, m.dNdX)
    A = O.tangent_A(m.qmat(O.Material("linear_elastic", E=1e3, nu=0.3)), F)
    K = O.assemble(O.element_stiffness(A, m.dNdX, m.vol), conn, v.n_nodes)
    free = sp.diags((~v.fixed_mask.reshape(-1)).astype(float))
    rhs = np.random.default_rng(3).standard_normal(v.X.shape)
    rhs[v.fixed_mask] = 0.0
    return request.param, v, (free @ K @ free).tocsr(), rhs.reshape(-1)


def _interpolation(X, conn, cell):
    """P: [3 nodes, 3 corners of the cells that hold an element's centre]."""
    h = 32.0 / N
    H = cell * h
    lo, hi = X.min(0), X.max(0)
    g = np.maximum(1, np.ceil((hi - lo) / H - 1e-9).astype(int))
    org = lo - np.floor(0.5 * (g * H - (hi - lo)) / h + 1e-6) * h
    ijk = np.clip(np.floor((X[conn].mean(1) - org) / H).astype(int), 0, g - 1)
    off = np.array([[q >> 2 & 1, q >> 1 & 1, q & 1] for q in range(8)])

    def lattice(c):
        c = c[:, None, :] + off[None]
        return (c[..., 0] * (g[1] + 1) + c[..., 1]) * (g[2] + 1) + c[..., 2]

    used = np.unique(lattice(ijk))
    # a node's cell: that of one of its elements (on a cell's face all give the same weights)
    cell_of = np.zeros(X.shape, dtype=int)
    for k in range(conn.shape[1]):
        cell_of[conn[:, k]] = ijk
    t = np.clip((X - org) / H - cell_of, 0.0, 1.0)
    w = np.prod(np.where(off[None] == 1, t[:, None, :], 1.0 - t[:, None, :]), axis=-1)
    cols = np.searchsorted(used, lattice(cell_of))
    P = sp.coo_matrix((w.ravel(), (np.repeat(np.arange(len(X)), 8), cols.ravel())), shape=(len(X), used.size)).tocsr()
    return sp.kron(P, sp.eye(3)).tocsr()


def _z(K, P, fixed, r, block):
    Ac = (P.T @ K @ P).tocsc()
    dead = Ac.diagonal() <= 1e-9 * Ac.diagonal().max()
    Ac = Ac + sp.diags(dead.astype(float))
    z = P @ spsolve(Ac.tocsc(), P.T @ r)
    if block:
        n = K.shape[0] // 3
        D = np.zeros((n, 3, 3))
        for i in range(3):
            for j in range(3):
                D[:, i, j] = K[3 * np.arange(n) + i, 3 * np.arange(n) + j]
        f = fixed.reshape(n, 3)
        D[f[:, :, None] | f[:, None, :]] = 0.0
        for i in range(3):
            D[f[:, i], i, i] = 1.0
        z += np.einsum("nij,nj->ni", np.linalg.inv(D), r.reshape(n, 3)).reshape(-1)
    else:
        d = K.diagonal()
        z += np.where(fixed.reshape(-1), 0.0, r / np.where(d > 0, d, 1.0))
    z[fixed.reshape(-1)] = 0.0
    return z


@pytest.mark.parametrize("variant", ["auto", "two_phase"])
@pytest.mark.parametrize("block", [True, False])
@pytest.mark.parametrize("cell", [2, 3, 4, 6, 12])
def test_first_iterate(cuda, body, cell, block, variant):
    element, v, K, r = body
    P = _interpolation(v.X, v.conn.astype(np.int64), cell)
    z = _z(K, P, v.fixed_mask, r, block)
    want = (r @ z) / (z @ (K @ z)) * z
    mesh = B.FEMesh(v.n_nodes, v.n_elements, B.ElementType.HEX8 if element == "hex8" else B.ElementType.TET4,
                    device=cuda)
    mesh.initialize_from_numpy(v.X, v.conn)
    mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
    B.LinearElastic(1e3, 0.3).compute_nodal_forces(mesh)
    mesh.set_coarse_options(cell=cell)
    mesh.set_block_smoother(block)
    mesh.set_matvec_variant(variant)
    dr = torch.from_numpy(r.reshape(-1, 3)).to(cuda)
    du = torch.zeros_like(dr)
    it, rel = C.c_int32(), C.c_double()
    rc = _lib.load().fem_pcg(mesh.ctx, _lib.FEM_PRECOND_TWO_LEVEL, B._ptr(dr), B._ptr(du), 1e-12, 1, C.byref(it),
                             C.byref(rel))
    assert rc == _lib.FEM_NOT_CONVERGED and it.value == 1, _lib.last_error(mesh.ctx)
    info = mesh.coarse_info()
    assert info["coarse_dofs"] == P.shape[1] and info["jacobi_fallbacks"] == 0
    assert np.linalg.norm(du.cpu().numpy().reshape(-1) - want) < 1e-3 * np.linalg.norm(want)
