"""FP64 residual whose elements are pipelined (history staged one element
ahead, slot forces as 32-byte rows): element counts around a block's 128 and
one where each resident thread takes several elements, TET4 and HEX8, with a
committed J2 history, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from oracle import fem_oracle as O
from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu

# FP64 on both sides; near the yield surface the return map's branch and its
# divisions may round differently
TOL = 1e-8


@pytest.mark.parametrize("kind,ne", [("tet4", 1), ("tet4", 127), ("tet4", 129), ("tet4", None), ("hex8", 1),
                                     ("hex8", 129), ("hex8", None)])
def test_pipelined_residual_matches_oracle(cuda, kind, ne):
    if kind == "tet4":
        bar = meshgen.cantilever_bar(nx=40, ny=23, nz=22) if ne is None else meshgen.cantilever_bar(nx=5, ny=3, nz=3)
        X, conn = bar.X, np.asarray(bar.conn)
    else:
        X, conn = meshgen.structured_hex8(7, 6, 6, (7.0, 6.0, 6.0))
    conn = conn[:ne]
    used = np.unique(conn)
    X, conn = X[used], np.searchsorted(used, conn).astype(np.int32)
    et = B.ElementType.HEX8 if kind == "hex8" else B.ElementType.TET4
    mesh = B.FEMesh(X.shape[0], conn.shape[0], et, device=cuda)
    mesh.initialize_from_numpy(X, conn)
    mat = B.J2Plasticity(1e3, 0.3, 5.0, hardening_modulus=20.0)
    om = O.Material("j2", E=1e3, nu=0.3, sigma_y=5.0, H=20.0)
    m = O.Mesh(X, conn)
    rng = np.random.default_rng(len(conn))
    u = 0.01 * rng.standard_normal(X.shape)
    mesh.u.copy_(torch.from_numpy(u))
    mat.compute_nodal_forces(mesh)
    want = O.internal_state(m, om, u)
    assert np.abs(mesh.get_nodal_forces() - want[3]).max() <= TOL * np.abs(want[3]).max()
    # from the committed history, at another displacement
    assert _lib.load().fem_commit_history(mesh.ctx) == 0
    state = want[4][0]
    u2 = u + 0.005 * rng.standard_normal(X.shape)
    mesh.u.copy_(torch.from_numpy(u2))
    mat.compute_nodal_forces(mesh)
    f2 = O.internal_state(m, om, u2, state)[3]
    assert np.abs(mesh.get_nodal_forces() - f2).max() <= TOL * np.abs(f2).max()
