"""The V-cycle's tiles, bottom levels and enrichment pieces at the grid sizes
where they begin, end and leave remainders, against the oracle's direct solve."""
import numpy as np
import pytest

import oracle
import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE, rsa_circles

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


# Enrichment pieces of cohesive meshes: 60 rows (64 thread groups suffice), 112
# (as many as the wide CTA has groups) and 160 (rows beyond them, in a loop).
# Newton to 1e-11 of the first residual, as for the other cohesive paths: 1e-7.
@pytest.mark.parametrize("nx,ny,circles", [(24, 24, [(0.5, 0.5, 0.3)]), (24, 20, (1, 16, 0.07, 0.1, 0.004)),
                                           (64, 64, (1, 250, 0.02, 0.03, 0.001))])
@pytest.mark.parametrize("precision", [_lib.PG_PRECISION_FP64, _lib.PG_PRECISION_MIXED])
def test_mg_cohesive_pieces_match_oracle_newton(nx, ny, circles, precision):
    if isinstance(circles, tuple):
        circles = rsa_circles(*circles, max_tries=20000)
    rve = RVE(nx=nx, ny=ny, inclusions=[(x, y, r, 1) for x, y, r in circles], cohesive=True, coh_law=1,
              coh_params=(30.0, 1.0, 1.0e6, 1.0), strain=0.001)
    prob = pb.ProblemNonlinearStructural(rve)
    prob.init()
    prob.configure(rtol=1e-11, precision=precision, precond=_lib.PG_PREC_MG)
    e = prob.mesh.export()
    om = oracle.from_product(e, pb.template_table(), rve)
    st = prob.load_step(0.5, 0.5)
    assert st.reason > 0, st.reason
    U, _, _, _, _ = oracle.newton_load_step(om, np.zeros(prob.mesh.info["n_dof"]), e["fixed"], e["ubar"], 0.5, 0.5,
                                            np.zeros(prob.mesh.info["n_cohesive_qp"]), rtol=1e-11)
    u = prob.get_solution()
    assert np.linalg.norm(u - U) / np.linalg.norm(U) <= 1e-7
    prob.ctx.close()
