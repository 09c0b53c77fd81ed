"""The tables of the assembled tangent, derived on the device: nodes with few and
with very many elements (the sorting warp's chunks of 32), unordered node and
element numbers, nodes without elements; against the FP64 oracle's direct solve
(FP32 vectors, residual to 1e-7: 1e-5 by the condition of these small systems)."""
import ctypes as C

import numpy as np
import pytest
import torch
from scipy.spatial import ConvexHull

from oracle import fem_oracle as O
from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu


def _solve(X, conn, fixed, hexa, cuda):
    """(solution of a random right-hand side, the oracle's, the variant taken, device bytes that the solve added)"""
    mesh = B.FEMesh(X.shape[0], conn.shape[0], B.ElementType.HEX8 if hexa else B.ElementType.TET4, device=cuda)
    mesh.initialize_from_numpy(X, conn)
    mesh.set_fixed_dofs(np.where(fixed.reshape(-1))[0])
    mat = B.LinearElastic(1e3, 0.3)
    mat.compute_nodal_forces(mesh)
    rhs = np.random.default_rng(1).standard_normal(X.shape)
    rhs[fixed] = 0.0
    r = torch.from_numpy(rhs).to(cuda)
    du = torch.zeros_like(r)
    before = mesh.info()["device_bytes"]
    it, rel = C.c_int32(), C.c_double()
    rc = _lib.load().fem_pcg(mesh.ctx, _lib.FEM_PRECOND_JACOBI, B._ptr(r), B._ptr(du), 1e-7, 20000, C.byref(it),
                             C.byref(rel))
    assert rc == 0, _lib.last_error(mesh.ctx)
    m = O.Mesh(X, conn)
    F = O.deformation_gradient(np.zeros_like(X), m.qconn if hexa else conn.astype(np.int64), m.dNdX)
    want = O.solve_tangent(O.Material("linear_elastic", E=1e3, nu=0.3), F, None, m, rhs, fixed)
    return du.cpu().numpy(), want, mesh.stats()["matvec_variant"], mesh.info()["device_bytes"] - before


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# tets between a centre and the triangles of a sphere: 30, 32, 34, 900, 8,096 and 9,996 elements on one node; the
# centre's row alone has too many pieces for the kernel's shared memory in the last but one, and the last is above
# what the tables take: both run as the kernel chain and keep no tables
@pytest.mark.parametrize("points", [17, 18, 19, 452, 4050, 5000])
def test_many_elements_on_one_node(cuda, points):
    k = np.arange(points) + 0.5
    polar, az = np.arccos(1.0 - 2.0 * k / points), np.pi * (1.0 + 5.0 ** 0.5) * k
    S = np.stack([np.cos(az) * np.sin(polar), np.sin(az) * np.sin(polar), np.cos(polar)], axis=1)
    X = np.concatenate([S, [[0.0, 0.0, 0.0]]])
    tri = ConvexHull(S).simplices
    n = np.cross(S[tri[:, 1]] - S[tri[:, 0]], S[tri[:, 2]] - S[tri[:, 0]])
    flip = np.einsum("ij,ij->i", n, S[tri].mean(1)) < 0.0
    tri[flip] = tri[flip][:, ::-1]
    conn = np.concatenate([np.full((len(tri), 1), points), tri], axis=1).astype(np.int32)
    fixed = np.zeros(X.shape, dtype=bool)
    fixed[:points:3] = True
    got, want, variant, added = _solve(X, conn, fixed, False, cuda)
    assert (variant == "assembled") == (points <= 452)
    assert (added > 0) == (variant == "assembled")
    assert _rel(got, want) < 1e-5


@pytest.mark.parametrize("element", ["tet4", "hex8"])
def test_unordered_numbers_and_nodes_without_elements(cuda, element):
    v = meshgen.vertebral_body(n=10, seed=1, element=element)
    rng = np.random.default_rng(0)
    nn = v.n_nodes + 7
    p = rng.permutation(nn)
    X = rng.uniform(-1.0, 1.0, (nn, 3))
    X[p[:v.n_nodes]] = v.X
    fixed = np.ones(X.shape, dtype=bool)
    fixed[p[:v.n_nodes]] = v.fixed_mask
    conn = p[v.conn][rng.permutation(v.n_elements)].astype(np.int32)
    got, want, variant, _ = _solve(X, conn, fixed, element == "hex8", cuda)
    assert variant == "assembled"
    assert _rel(got, want) < 1e-5
