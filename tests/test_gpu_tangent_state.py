"""The assembled blocks follow the tangent payload: a solve uses the blocks of
the payload that the element product (``fem_tangent_matvec``) uses."""
import ctypes as C

import numpy as np
import pytest
import torch

from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu


def _plastic_body(cuda, element, n=8):
    """A J2 body compressed past yield, forces evaluated there."""
    v = meshgen.vertebral_body(n=n, element=element)
    mesh = B.FEMesh(v.n_nodes, v.n_elements, B.ElementType.HEX8 if element == "hex8" else B.ElementType.TET4,
                    device=cuda)
    mesh.initialize_from_numpy(v.X, v.conn)
    mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
    mat = B.J2Plasticity(v.E, 0.3, 100.0, hardening_modulus=0.02 * v.E)
    u = np.zeros_like(v.X)
    u[:, 2] = -0.03 * v.X[:, 2]
    mesh.u.copy_(torch.from_numpy(u))
    mat.compute_nodal_forces(mesh)
    rhs = np.random.default_rng(1).standard_normal(v.X.shape)
    rhs[v.fixed_mask] = 0.0
    return mesh, mat, torch.from_numpy(rhs).to(cuda)


def _solve(mesh, r, pc=_lib.FEM_PRECOND_TWO_LEVEL, rtol=1e-7):
    du = torch.zeros_like(r)
    it, rel = C.c_int32(), C.c_double()
    rc = _lib.load().fem_pcg(mesh.ctx, pc, B._ptr(r), B._ptr(du), rtol, 20000, C.byref(it), C.byref(rel))
    assert rc == 0, _lib.last_error(mesh.ctx)
    return du


def _residual(mesh, du, r):
    """||K du - r|| / ||r|| with the element product."""
    x = du.to(torch.float32)
    y = torch.empty_like(x)
    assert _lib.load().fem_tangent_matvec(mesh.ctx, B._ptr(x), B._ptr(y)) == 0
    return float((y.double() - r).norm() / r.norm())


# FP32 products and a residual of 1e-7 by recurrence leave 1e-4 at most on these small systems
@pytest.mark.parametrize("element", ["tet4", "hex8"])
def test_solve_after_profiling_uses_the_new_tangent(cuda, element):
    mesh, _, r = _plastic_body(cuda, element)
    lib = _lib.load()
    assert _residual(mesh, _solve(mesh, r), r) < 1e-4
    # the committed state lies on the yield surface: the tangent evaluated
    # again at the same u, by the profiling call, is the elastic one there
    assert lib.fem_commit_history(mesh.ctx) == 0
    ms = (C.c_double * 4)()
    assert lib.fem_profile_kernels(mesh.ctx, 1, ms) == 0
    assert _residual(mesh, _solve(mesh, r), r) < 1e-4


def test_network_output_does_not_depend_on_an_earlier_solve(cuda):
    from simul_b200 import learned
    mesh, _, r = _plastic_body(cuda, "tet4")
    learned.set_weights(mesh, learned.init_weights(seed=2, out_scale=0.2))
    x = r.to(torch.float32)
    z = []
    for solve_first in (False, True):
        if solve_first:
            _solve(mesh, r)
            assert mesh.stats()["matvec_variant"] == "assembled"
        z.append(torch.empty_like(x))
        assert _lib.load().fem_mpnn_forward(mesh.ctx, B._ptr(x), B._ptr(z[-1])) == 0
    assert torch.equal(z[0], z[1])
