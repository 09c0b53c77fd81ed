"""The coarse operator's cells in chunks of 32 elements: bodies whose lattice
cells hold a few to several hundred elements (remainders of a chunk, several
chunks, several slices).  A wrong block shows in the iteration count of the
two-level solve, which the entry-by-entry assembly of an earlier version fixed
(one iteration for the different association of the FP64 sums)."""
import ctypes as C

import numpy as np
import pytest
import torch

from simul_b200 import _lib, meshgen
from simul_b200 import fem as B

pytestmark = pytest.mark.gpu

# cell size in voxels -> iterations with the block and with the diagonal smoother
COUNTS = {1: (12, 12), 2: (28, 28), 3: (38, 40), 4: (47, 48), 6: (55, 56), 8: (59, 61), 16: (91, 93)}


@pytest.mark.parametrize("cell", sorted(COUNTS))
@pytest.mark.parametrize("block", [True, False])
def test_two_level_iterations_by_cell_size(cuda, cell, block):
    v = meshgen.vertebral_body(n=16, seed=3)
    mesh = B.FEMesh(v.n_nodes, v.n_elements, device=cuda)
    mesh.initialize_from_numpy(v.X, v.conn)
    mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
    mat = B.LinearElastic(v.E, 0.3)
    mat.compute_nodal_forces(mesh)
    mesh.set_coarse_options(cell=cell)
    mesh.set_block_smoother(block)
    rhs = np.random.default_rng(3).standard_normal(v.fixed_mask.shape)
    rhs[v.fixed_mask] = 0.0
    r = torch.from_numpy(rhs).to(cuda)
    du = torch.zeros_like(r)
    it, rel = C.c_int32(), C.c_double()
    rc = _lib.load().fem_pcg(mesh.ctx, _lib.FEM_PRECOND_TWO_LEVEL, B._ptr(r), B._ptr(du), 1e-6, 2000, C.byref(it),
                             C.byref(rel))
    assert rc == 0, _lib.last_error(mesh.ctx)
    assert abs(it.value - COUNTS[cell][0 if block else 1]) <= 1
