"""Stress outputs whose rows are turned in shared memory, and the nodal von
Mises pass through the slot staging: element counts around a warp's 32 rows
and a block's 128, TET4 and HEX8, with F and the stress wanted together or
one of them alone, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from oracle import fem_oracle as O
from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu

# FP64 evaluation of the same expressions: a few hundred roundings of 1.1e-16
# on strains of size 0.1, cancellation against the identity allowed for
TOL = 1e-11


def _meshes():
    X, conn = meshgen.structured_hex8(5, 5, 6, (5.0, 5.0, 6.0))
    tets = np.asarray(meshgen.cantilever_bar(nx=5, ny=3, nz=3).conn)
    bar = meshgen.cantilever_bar(nx=5, ny=3, nz=3)
    for ne in (1, 31, 32, 33, 127, 128, 129, tets.shape[0]):
        yield "tet4", bar.X, tets[:ne]
    for ne in (1, 33, 128, 129, conn.shape[0]):
        yield "hex8", X, conn[:ne]


@pytest.mark.parametrize("case", list(_meshes()), ids=lambda c: f"{c[0]}-{len(c[2])}")
def test_rows_and_nodal_sums_match_oracle(cuda, case):
    kind, X, conn = case
    used = np.unique(conn)
    X, conn = X[used], np.searchsorted(used, conn).astype(np.int32)
    et = B.ElementType.HEX8 if kind == "hex8" else B.ElementType.TET4
    mesh = B.FEMesh(X.shape[0], conn.shape[0], et, device=cuda)
    mesh.initialize_from_numpy(X, conn)
    u = 0.02 * np.random.default_rng(len(conn)).standard_normal(X.shape)
    mesh.u.copy_(torch.from_numpy(u))
    mat = B.NeoHookean(17e3, 0.3)
    om = O.Material("neo_hookean", E=17e3, nu=0.3)
    m = O.Mesh(X, conn)
    F, sigma = O.internal_state(m, om, u)[:2]
    mat.compute_stress(mesh)
    got_F, got_s = mesh.F.clone(), mesh.stress.clone()
    assert np.abs(got_F.cpu().numpy().reshape(F.shape) - F).max() <= TOL * np.abs(F).max()
    assert np.abs(got_s.cpu().numpy().reshape(sigma.shape) - sigma).max() <= TOL * np.abs(sigma).max()
    lib = _lib.load()
    one = torch.full_like(got_F, -7.0)
    assert lib.fem_compute_stress(mesh.ctx, None, B._ptr(one), None) == 0
    assert torch.equal(one, got_F)
    assert lib.fem_compute_stress(mesh.ctx, None, None, B._ptr(one)) == 0
    assert torch.equal(one, got_s)
    for average in (False, True):
        mesh.compute_mises_stress(average=average)
        want = O.nodal_mises(m, om, u, average=average)
        assert np.abs(mesh.mises.cpu().numpy() - want).max() <= TOL * np.abs(want).max()
