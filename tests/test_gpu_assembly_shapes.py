"""The structured-grid assembly kernels against the row-tile kernel, which
makes no use of the grid: every mode (stiffness, residual, both), sizes below,
at and above a tile, and more tiles than the GPU holds at once (the persistent
kernel), with cohesive and plain cut elements.

Both sum at most 8 triangles and 12 cut elements per value in another order: a
relative difference of 20 roundings (2.2e-15), and up to a factor 40 between
the norm of the summed terms and of the sum, stays below 1e-13."""
import numpy as np
import pytest

import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(12, 9), (64, 31), (63, 33), (65, 30), (129, 62), (640, 181)])
@pytest.mark.parametrize("law", [None, 0, 1])
def test_grid_kernels_agree_with_the_row_tiles(nx, ny, law):
    # two interfaces close together: cut elements of several size classes
    more = {} if law is None else dict(cohesive=True, coh_law=law, coh_params=(30.0, 0.01, 1.0, 0.5, 0.0) if law == 0
                                       else (30.0, 1.0, 1.0e6, 1.0, 0.0))
    rve = RVE(nx=nx, ny=ny, inclusions=[(0.28, 0.5, 0.2, 1), (0.74, 0.5, 0.21, 1)], strain=0.01, **more)
    m = pb.Mesh(rve)
    ctx = pb.DeviceContext(m)
    rng = np.random.default_rng(nx)
    ctx.set_vector(0, 1e-3 * rng.standard_normal(m.info["n_dof"]))
    if m.info["n_cohesive_qp"]:
        ctx.set_isv(np.abs(1e-3 * rng.standard_normal(m.info["n_cohesive_qp"])), committed=True)
    asm = pb.Assembler(ctx)

    def passes():
        got = []
        for f, K in ((True, True), (False, True), (True, False)):
            asm.assemble_nonlinear(0.02, f, K)
            got += [ctx.matrix_values().ravel()] * K + [ctx.vector(1)] * f
        return got + ([ctx.isv(committed=False)] if m.info["n_cohesive_qp"] else [])

    _lib.check(_lib.lib.pg_ctx_set_tuning(ctx.handle, 64, 0, 4))
    want = passes()
    for tile in (128, 256):
        for persistent in (0, 1):
            _lib.check(_lib.lib.pg_ctx_set_tuning(ctx.handle, tile, persistent, 4))
            got = passes()
            for g, w in zip(got, want):
                assert np.linalg.norm(g - w) <= 1e-13 * np.linalg.norm(w)
            assert all(np.array_equal(a, b) for a, b in zip(got, passes()))
    ctx.close()
