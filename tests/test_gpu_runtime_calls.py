"""What the library asks of the CUDA runtime, seen by a stand-in in front of it."""
import pytest

import cudart_shim

pytestmark = pytest.mark.gpu


def test_an_explicit_launch_shape_is_the_one_that_runs(tmp_path):
    # a mesh whose grid tiles fit the GPU all at once: by default one CTA per
    # tile, but persistent 0 and 1 launch their own kernels, and what is read
    # back sets the same again
    cudart_shim.run(tmp_path, r"""
ctx = pb.DeviceContext(pb.Mesh(RVE(nx=40, ny=30, strain=0.01)))
asm = pb.Assembler(ctx)
def one(tile, persistent):
    _lib.check(_lib.lib.pg_ctx_set_tuning(ctx.handle, tile, persistent, 4))
    return kernels(asm.assemble_linear)
tile, persistent, warps = C.c_int32(), C.c_int32(), C.c_int32()
_lib.check(_lib.lib.pg_ctx_tuning(ctx.handle, C.byref(tile), C.byref(persistent), C.byref(warps)))
default = kernels(asm.assemble_linear)
assert one(tile.value, persistent.value) == default
assert (tile.value, persistent.value) == (128, 0)
for t in (128, 256):
    assert one(t, 0) != one(t, 1), t
ctx.close()
""")


def test_function_attributes_do_not_depend_on_the_context(tmp_path):
    # they belong to the device: a value of one context's own size could be
    # lowered by another host thread before the launch that needs it
    cudart_shim.run(tmp_path, r"""
crowded = [(i / 12, j / 12, 0.42 / 12, 1) for j in range(13) for i in range(13)]
for precision in (_lib.PG_PRECISION_FP64, _lib.PG_PRECISION_MIXED):
    for precond in (_lib.PG_PREC_BLOCK_JACOBI, _lib.PG_PREC_MG):
        for nx, inclusions in ((12, crowded), (40, [(0.5, 0.5, 0.25, 1)]), (100, [(0.5, 0.5, 0.25, 1)])):
            prob = pb.ProblemLinearElasticity(RVE(nx=nx, ny=nx, inclusions=inclusions, strain=0.01))
            prob.init()
            for warps in (2, 4, 8):
                _lib.check(_lib.lib.pg_ctx_set_tuning(prob.ctx.handle, 128, 0, warps))
                pb.Assembler(prob.ctx).assemble_linear()
            prob.get_solver().configure(precond=precond, precision=precision, rtol=1e-9)
            prob.solve_problem()
            prob.ctx.close()
n = var("shim_n_attr").value
funcs, attrs, values = (var(name, k * 65536) for name, k in
                        (("shim_attr_func", C.c_void_p), ("shim_attr", C.c_int), ("shim_attr_value", C.c_int)))
seen = {}
for i in range(n):
    seen.setdefault((funcs[i], attrs[i]), set()).add(values[i])
assert len(seen) > 8, seen
assert all(len(v) == 1 for v in seen.values()), seen
""")


def test_a_refused_launch_ends_the_multigrid_solve_and_no_later_one(tmp_path):
    # refused while a V-cycle is queued, or while the iterations are recorded:
    # an error there and then, and the next solve is that of a fresh context
    cudart_shim.run(tmp_path, r"""
def problem():
    prob = pb.ProblemLinearElasticity(RVE(nx=48, ny=40, inclusions=[(0.5, 0.5, 0.27, 1)], strain=0.01))
    prob.init()
    prob.get_assembler().assemble_linear()
    return prob
def solve(prob, precision):
    s = prob.get_solver()
    s.configure(precond=_lib.PG_PREC_MG, precision=precision, rtol=1e-10, max_iter=300)
    prob.ctx.set_vector(0, np.zeros(prob.mesh.info["n_dof"]))
    return _lib.lib.pg_solve_linear(prob.ctx.handle, C.byref(s.cfg), C.byref(s.stats))
for precision in (_lib.PG_PRECISION_FP64, _lib.PG_PRECISION_MIXED):
    clean = problem()
    assert solve(clean, precision) == 0
    for captured in (0, 1):
        for nth in range(0, 8):  # fewer than a cycle's launches
            prob = problem()
            var("shim_refuse_captured").value = captured
            var("shim_refuse").value = nth
            rc = solve(prob, precision)
            assert var("shim_refuse").value == -1
            assert rc == _lib.PG_ERR_CUDA, (captured, nth, rc)
            assert solve(prob, precision) == 0, (captured, nth)
            assert np.array_equal(prob.get_solution(), clean.get_solution()), (captured, nth)
            prob.ctx.close()
""")
