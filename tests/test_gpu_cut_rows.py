"""The cut elements' quadrature rows are formed in two ways: straight from the
point records in a stiffness pass, and from node coordinates staged for the
whole CTA where the pass has displacements too.  Both evaluate the same
expressions at the same coordinates; the stiffness may differ by the
contraction of its sums alone (at most 27 points and 8 triangles per value, a
factor 40 between the norm of the terms and of the sum: 1e-13)."""
import numpy as np
import pytest

import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE

pytestmark = pytest.mark.gpu


def _crowded(n):
    """A circle around every node: each element is cut on its three sides."""
    return [(i / n, j / n, (0.45 if (i + j) % 2 == 0 else 0.4) / n, 1) for j in range(n + 1) for i in range(n + 1)]


@pytest.mark.parametrize("nx,ny,inclusions", [
    (5, 4, [(0.5, 0.5, 0.21, 1)]),                                  # fewer elements than a CTA takes
    (64, 31, [(0.28, 0.5, 0.2, 1), (0.74, 0.5, 0.21, 1)]),          # elements of two and four enrichment nodes
    (12, 12, _crowded(12)),                                         # six, with children of six sides
    (40, 40, _crowded(40)),                                         # and more than one point per thread
])
@pytest.mark.parametrize("warps", [2, 4, 8])
def test_both_ways_to_form_the_rows_give_the_same_stiffness(nx, ny, inclusions, warps):
    ctx = pb.DeviceContext(pb.Mesh(RVE(nx=nx, ny=ny, inclusions=inclusions, strain=0.01)))
    ctx.set_vector(0, 1e-3 * np.random.default_rng(nx).standard_normal(ctx.info["n_dof"]))
    _lib.check(_lib.lib.pg_ctx_set_tuning(ctx.handle, 128, 0, warps))
    asm = pb.Assembler(ctx)
    asm.assemble_nonlinear(0.02, True, True)
    staged = ctx.matrix_values()
    for _ in range(2):
        asm.assemble_nonlinear(0.02, False, True)
        K = ctx.matrix_values()
        assert np.linalg.norm(K - staged) <= 1e-13 * np.linalg.norm(staged)
    ctx.close()
