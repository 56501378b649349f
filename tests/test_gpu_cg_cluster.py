"""Block-Jacobi and Jacobi CG at the sizes where its one-launch form changes:
fewer rows than CTAs, blocks of K in shared memory, blocks in global memory,
and too large for it; against the oracle's direct solve."""
import numpy as np
import pytest

import oracle
import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,circle", [(1, 2, False), (3, 3, False), (16, 15, True), (64, 64, True), (90, 90, True),
                                          (97, 101, True), (150, 130, True), (170, 171, True)])
@pytest.mark.parametrize("precond", [_lib.PG_PREC_BLOCK_JACOBI, _lib.PG_PREC_JACOBI])
def test_cg_matches_direct_solve(nx, ny, circle, precond):
    rve = RVE(nx=nx, ny=ny, inclusions=[(0.5, 0.48, 0.27, 1)] if circle else [], strain=0.01)
    prob = pb.ProblemLinearElasticity(rve)
    prob.init()
    e = prob.mesh.export()
    prob.get_solver().configure(precond=precond, rtol=1e-11)
    runs = []
    for _ in range(2):
        prob.ctx.set_vector(0, np.zeros(prob.mesh.info["n_dof"]))
        st = prob.solve_problem()
        assert st.status == 0, st.status
        runs.append(prob.get_solution())
    assert np.array_equal(runs[0], runs[1])
    Ko, _, _ = oracle.from_product(e, pb.template_table(), rve).assemble()
    uo = oracle.solve_linear(Ko, e["fixed"], e["ubar"])
    assert np.linalg.norm(runs[0] - uo) / np.linalg.norm(uo) <= 1e-8
    prob.ctx.close()


def test_cg_budget_is_honoured_exactly():
    prob = pb.ProblemLinearElasticity(RVE(nx=32, ny=32, strain=0.01))
    prob.init()
    prob.get_solver().configure(rtol=1e-12, max_iter=7)
    with pytest.raises(_lib.PgError):
        prob.solve_problem()
    assert prob.get_solver().stats.iterations == 7
    prob.ctx.close()


@pytest.mark.parametrize("nx,ny,circle", [(1, 2, False), (16, 15, True), (64, 64, True), (110, 112, True), (116, 118, True),
                                          (150, 130, True), (170, 171, True)])
@pytest.mark.parametrize("precond", [_lib.PG_PREC_BLOCK_JACOBI, _lib.PG_PREC_JACOBI])
def test_mixed_precision_reaches_the_residual_it_is_asked_for(nx, ny, circle, precond):
    """K stored in FP32: its blocks fit shared memory up to 110 x 112, the rest of the system up to 150 x 130;
    beyond, launches.  The refinement ends by the FP64 residual, so that of the oracle's matrix is at most rtol,
    plus the rounding of both products: at most 40 products and sums in a row, 50 u |K| |u| with a margin."""
    rve = RVE(nx=nx, ny=ny, inclusions=[(0.5, 0.48, 0.27, 1)] if circle else [], strain=0.01)
    prob = pb.ProblemLinearElasticity(rve)
    prob.init()
    e = prob.mesh.export()
    rtol = 1e-11
    prob.get_solver().configure(precond=precond, precision=_lib.PG_PRECISION_MIXED, rtol=rtol)
    runs = []
    for _ in range(2):
        prob.ctx.set_vector(0, np.zeros(prob.mesh.info["n_dof"]))
        st = prob.solve_problem()
        assert st.status == 0, st.status
        runs.append(prob.get_solution())
    assert np.array_equal(runs[0], runs[1])
    Ko, _, _ = oracle.from_product(e, pb.template_table(), rve).assemble()
    free = ~np.asarray(e["fixed"], bool)
    u = runs[0]
    b = np.linalg.norm((Ko @ np.where(free, 0.0, e["ubar"]))[free])
    rounding = 50 * 2.0 ** -53 * np.linalg.norm((abs(Ko) @ abs(u))[free])
    assert np.array_equal(u[~free], np.asarray(e["ubar"])[~free])
    assert np.linalg.norm((Ko @ u)[free]) <= rtol * b + 2 * rounding
    prob.ctx.close()
