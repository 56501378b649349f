"""A context keeps what its sensitivities need; calls in any order, with other
parameters, another state and the finite-difference form between them, give
what the first call of a new context gives.

The element derivatives are summed with atomics, n terms per parameter in any
order, and the adjoint solve starts from the same data: 1e-10 of the largest
derivative is far above both roundings and far below any stale input."""
import ctypes as C

import numpy as np
import pytest

import pigfem_assignment_b200.problem as pb
from pigfem_assignment_b200 import _lib
from pigfem_assignment_b200.rve import RVE

pytestmark = pytest.mark.gpu


def config():
    cfg = _lib.SolverCfg()
    _lib.lib.pg_solver_cfg_default(C.byref(cfg))
    cfg.precond, cfg.rtol, cfg.max_iter = _lib.PG_PREC_MG, 1e-12, 10000
    return cfg


def problem(U=None):
    prob = pb.ProblemLinearElasticity(RVE(nx=37, ny=29, inclusions=[(0.3, 0.5, 0.18, 1), (0.72, 0.4, 0.14, 1)], strain=0.01))
    prob.init()
    prob.get_solver().configure(precond=_lib.PG_PREC_MG, rtol=1e-12)
    prob.solve_problem()
    if U is not None:
        prob.ctx.set_vector(0, U)
    return prob


def shape(prob, params):
    inc = np.array([p[0] for p in params], np.int32)
    kind = np.array([p[1] for p in params], np.int32)
    f, g = C.c_double(), np.zeros(len(params))
    _lib.check(_lib.lib.pg_sensitivity_shape(prob.ctx.handle, C.byref(config()), len(params), _lib.iptr(inc), _lib.iptr(kind),
                                             C.byref(f), _lib.dptr(g), None))
    return np.append(g, f.value)


def c11(prob, h):
    v, g = C.c_double(), np.zeros(2)
    _lib.check(_lib.lib.pg_sensitivity_c11(prob.ctx.handle, C.byref(config()), h, C.byref(v), _lib.dptr(g), None))
    return np.append(g, v.value)


X, Y, R = _lib.PG_SHAPE_X, _lib.PG_SHAPE_Y, _lib.PG_SHAPE_R
CALLS = [lambda p: shape(p, [(0, X), (1, R), (0, Y)]), lambda p: c11(p, 1e-5), lambda p: shape(p, [(1, R), (1, R)]),
         lambda p: c11(p, 0.0), lambda p: shape(p, []), lambda p: shape(p, [(k, d) for k in (1, 0) for d in (R, Y, X)])]


def test_calls_of_one_context_are_those_of_new_ones():
    kept = problem()
    U = np.random.default_rng(3).standard_normal(kept.ctx.vector(0).size) * 1e-3
    for state in (None, U):
        if state is not None:
            kept.ctx.set_vector(0, state)
        for call in CALLS:
            new = problem(state)
            want, got = call(new), call(kept)
            np.testing.assert_allclose(got, want, rtol=0, atol=1e-10 * np.abs(want).max())
            new.ctx.close()
    kept.ctx.close()
