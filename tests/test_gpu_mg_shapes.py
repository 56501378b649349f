"""The V-cycle's tiles, bottom levels and enrichment pieces at the grid sizes
where they begin, end and leave remainders, against the oracle's direct solve."""
import numpy as np
import pytest

import oracle
import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE

pytestmark = pytest.mark.gpu

ONE = [(0.47, 0.52, 0.23, 1)]
FOUR = [(0.3, 0.3, 0.13, 1), (0.72, 0.31, 0.16, 1), (0.29, 0.73, 0.17, 1), (0.71, 0.7, 0.11, 1)]


# (5, 5): the coarsest grid alone below level 0; (31, 31), (33, 33): level 1 of
# 16 and 17 cells, the last that the bottom takes whole; (35, 34): one cell
# more, so a tiled level of 18 x 17 cells; (70, 37): ragged tiles at every
# level; (6, 200), (200, 6): a side that stops halving early
@pytest.mark.parametrize("nx,ny,inclusions", [(5, 5, []), (31, 31, ONE), (33, 33, ONE), (35, 34, ONE), (70, 37, FOUR),
                                              (6, 200, []), (200, 6, []), (47, 90, FOUR)])
@pytest.mark.parametrize("precision", [_lib.PG_PRECISION_FP64, _lib.PG_PRECISION_MIXED])
def test_mg_solve_matches_direct_solve(nx, ny, inclusions, precision):
    rve = RVE(nx=nx, ny=ny, inclusions=list(inclusions), strain=0.01)
    prob = pb.ProblemLinearElasticity(rve)
    prob.init()
    e = prob.mesh.export()
    prob.get_solver().configure(precision=precision, precond=_lib.PG_PREC_MG, rtol=1e-12)
    st = prob.solve_problem()
    assert st.status == 0, st.status
    Ko, _, _ = oracle.from_product(e, pb.template_table(), rve).assemble()
    uo = oracle.solve_linear(Ko, e["fixed"], e["ubar"])
    u = prob.get_solution()
    assert np.linalg.norm(u - uo) / np.linalg.norm(uo) <= 1e-8
    prob.ctx.close()
