"""Which way a solve takes: the persistent kernel on the assembled tangent by
default, the kernel chain where an option asks for it, and back."""
import ctypes as C

import numpy as np
import pytest
import torch

from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu


class System:
    def __init__(self, cuda, element="tet4", n=8):
        v = meshgen.vertebral_body(n=n, element=element)
        self.mesh = B.FEMesh(v.n_nodes, v.n_elements,
                             B.ElementType.HEX8 if element == "hex8" else B.ElementType.TET4, device=cuda)
        self.mesh.initialize_from_numpy(v.X, v.conn)
        self.mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
        self.mat = B.LinearElastic(v.E, 0.3)
        self.mat.compute_nodal_forces(self.mesh)
        rhs = np.random.default_rng(1).standard_normal(v.X.shape)
        rhs[v.fixed_mask] = 0.0
        self.r = torch.from_numpy(rhs).to(cuda)

    def variant(self, pc=_lib.FEM_PRECOND_TWO_LEVEL):
        """The variant that a solve takes."""
        du = torch.zeros_like(self.r)
        it, rel = C.c_int32(), C.c_double()
        rc = _lib.load().fem_pcg(self.mesh.ctx, pc, B._ptr(self.r), B._ptr(du), 1e-6, 20000, C.byref(it), C.byref(rel))
        assert rc == 0, _lib.last_error(self.mesh.ctx)
        return self.mesh.stats()["matvec_variant"]


@pytest.mark.parametrize("element", ["tet4", "hex8"])
def test_options_at_their_defaults_keep_the_default_route(cuda, element):
    s = System(cuda, element)
    s.mesh.set_fused_step(False)
    s.mesh.set_whole_solve_graph(True)
    s.mesh.set_direction_recurrence(True)
    assert s.variant() == "assembled"
    for setter in (s.mesh.set_whole_solve_graph, s.mesh.set_direction_recurrence):
        setter(False)
        assert s.variant() != "assembled"
        setter(True)
        assert s.variant() == "assembled"


@pytest.mark.parametrize("element", ["tet4", "hex8"])
def test_the_rule_can_be_restored(cuda, element):
    s = System(cuda, element)
    asks = [lambda: s.mesh.set_programmatic_launch(True), lambda: s.mesh.set_matvec_variant("two_phase")]
    if element == "tet4":
        asks += [lambda: s.mesh.set_matvec_variant("fused"), lambda: s.mesh.set_matvec_variant(None)]
    for ask in asks:
        ask()
        assert s.variant() != "assembled"
        s.mesh.set_matvec_variant("auto")
        assert s.variant() == "assembled"
    s.mesh.set_fused_step(True)
    s.mesh.set_fused_step(False)
    assert s.variant() != "assembled"      # what was asked for stays
    s.mesh.set_matvec_variant("auto")
    assert s.variant() == "assembled"
    assert _lib.load().fem_set_option(s.mesh.ctx, _lib.FEM_OPT_MATVEC_VARIANT, -3) == _lib.FEM_ERR_INVALID


@pytest.mark.parametrize("grid,variant", [((7, 3, 3), "fused"), ((7, 3, 4), "persistent")])
def test_single_product_by_size(cuda, grid, variant):
    """128 nodes and 160: one launch, or the pair."""
    X, conn = meshgen.structured_tets(*grid)
    X = X + 0.02 / max(grid) * np.random.default_rng(0).standard_normal(X.shape)
    assert (X.shape[0] <= 128) == (variant == "fused")
    mesh = B.FEMesh(X.shape[0], conn.shape[0], device=cuda)
    mesh.initialize_from_numpy(X, conn)
    mat = B.NeoHookean(17e3, 0.3)
    mesh.u.copy_(torch.from_numpy(0.01 * np.random.default_rng(1).standard_normal(X.shape)))
    mat.compute_nodal_forces(mesh)
    x = torch.randn(X.shape, device=cuda, generator=torch.Generator(cuda).manual_seed(0))
    y = {}
    for v in ("auto", "fused", "persistent"):
        mesh.set_matvec_variant(v)
        y[v] = torch.empty_like(x)
        assert _lib.load().fem_tangent_matvec(mesh.ctx, B._ptr(x), B._ptr(y[v])) == 0
    assert not torch.equal(y["fused"], y["persistent"])   # told apart by rounding
    assert float((y["fused"] - y["persistent"]).norm() / y["fused"].norm()) < 1e-6
    assert torch.equal(y["auto"], y[variant])
