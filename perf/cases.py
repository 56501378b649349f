"""What a user of the framework has it do, as cases to be timed and compared.

Each case is one call (or the few calls) of a program that already holds its
meshes, device contexts or networks: the assembly of a linear RVE, the
residual and tangent of a cohesive one, linear solves, load stepping, a batch
of RVEs, the shape sensitivity, and the network of the learned start.  Sizes
follow the benchmark configurations (64^2, 256^2, 512^2 and 1024^2 background
meshes, 1 to 400 inclusions, batches of uneven RVEs) with ragged ones among
them.  Solves run to the tolerances at which their displacements are good to
about ten digits, the ones the parity tests use.
"""
import ctypes as C
import math

import numpy as np
import torch

from pigfem_assignment_b200 import _lib, learned, problem
from pigfem_assignment_b200.rve import COH_BILINEAR, COH_OP, RVE, rsa_circles

DEV = "cuda:0"
F64 = torch.float64


def listed():
    return [
        # the smallest RVE: one circle in 64x64, assembled alone (launch latency counts)
        dict(name="assemble_64", op="assemble", geometry=0, nx=64, ny=64, inc=1),
        # the benchmark's linear assembly pass: 512x512, 100 circles
        dict(name="assemble_512", op="assemble", geometry=1, nx=512, ny=512, inc=100),
        # residual and tangent of one Newton iteration, Ortiz-Pandolfi law, ragged grid
        dict(name="tangent_op_250x190", op="tangent", geometry=2, nx=250, ny=190, inc=23, law=COH_OP),
        # the same for the largest configuration: 1024x1024, 400 circles, bilinear law
        dict(name="tangent_1024", op="tangent", geometry=4, nx=1024, ny=1024, inc=400, law=COH_BILINEAR),
        # a small linear problem with the solver's default settings (block-Jacobi CG)
        dict(name="solve_default_64", op="solve", geometry=0, nx=64, ny=64, inc=1, mg=False, mixed=False, rtol=1e-12),
        # one linear load step of the benchmark RVE, FP64 multigrid
        dict(name="solve_512_fp64", op="solve", geometry=1, nx=512, ny=512, inc=100, mg=True, mixed=False, rtol=1e-12),
        # a large ragged one, FP32 multigrid cycle under the FP64 solve
        dict(name="solve_1000x700_mixed", op="solve", geometry=5, nx=1000, ny=700, inc=270, mg=True, mixed=True,
             rtol=1e-12),
        # load stepping of a cohesive RVE into the softening range, linear start, FP32 cycle
        dict(name="newton_256_mixed", op="newton", geometry=2, nx=256, ny=256, inc=40, steps=5, strain=0.01,
             mixed=True),
        # a batch of uneven RVEs (sides 64 to 256, 1 to 64 circles each), assembled and solved together
        dict(name="batch_32", op="batch", geometry=3, count=32, side=256, mixed=True, rtol=1e-12),
        # derivative of C_11 with respect to every radius: adjoint solve and element derivatives
        dict(name="sensitivity_256", op="sensitivity", geometry=2, nx=256, ny=256, inc=40, rtol=1e-12),
        # the learned start's network over the nodes of the largest configuration
        dict(name="mlp_forward_1m", op="mlp_forward", rows=1130000),
        # one epoch of its training in the benchmark's batches, the last one ragged
        dict(name="mlp_train_120k", op="mlp_train", rows=120000, batch=8192),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("assemble", "tangent", "solve", "newton", "batch", "sensitivity", "mlp_forward", "mlp_train"))
    if op == "mlp_forward":
        return dict(op=op, rows=_side(rng, 500, 1130000))
    if op == "mlp_train":
        return dict(op=op, rows=_side(rng, 1000, 120000), batch=_side(rng, 1000, 8192))
    geometry = rng.randint(10, 9999)
    if op == "batch":
        return dict(op=op, geometry=geometry, count=rng.randint(2, 32), side=rng.choice((96, 128, 192, 256)),
                    mixed=rng.random() < 0.5, rtol=1e-12)
    hi = dict(assemble=1024, tangent=1024, solve=700, newton=200, sensitivity=256)[op]
    nx, ny = _side(rng, 40, hi), _side(rng, 40, hi)
    inc = max(1, min(400, int(nx * ny / 2600.0 * rng.uniform(0.3, 1.2))))
    case = dict(op=op, geometry=geometry, nx=nx, ny=ny, inc=inc)
    if op == "tangent":
        case["law"] = rng.choice((COH_OP, COH_BILINEAR))
    elif op == "solve":
        case.update(mg=nx * ny > 20000 or rng.random() < 0.5, mixed=False, rtol=1e-12)
        case["mixed"] = case["mg"] and rng.random() < 0.5
    elif op == "newton":
        case.update(steps=rng.randint(2, 5), strain=round(rng.uniform(0.004, 0.01), 4), mixed=rng.random() < 0.5)
    elif op == "sensitivity":
        case["rtol"] = 1e-12
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rve(nx, ny, inc, geometry, seed, **more):
    """Circles at the area fraction of the benchmark configurations (radii 0.2 to 0.4 over sqrt(count)), placed by
    `geometry`; the materials, and with them the system to solve, are the seed's."""
    gap = max(0.005, 2.5 / min(nx, ny))
    n = inc
    while True:
        try:
            circ = rsa_circles(geometry, n, 0.2 / math.sqrt(n), min(0.4 / math.sqrt(n), 0.3), gap, max_tries=20000)
            break
        except RuntimeError:
            n = max(1, n // 2)
    g = np.random.default_rng(seed)
    materials = [(float(g.uniform(2500.0, 3500.0)), float(g.uniform(0.3, 0.38))),
                 (float(g.uniform(20000.0, 100000.0)), float(g.uniform(0.18, 0.25)))]
    return RVE(nx=nx, ny=ny, inclusions=[(x, y, r, 1) for (x, y, r) in circ], materials=materials, seed=geometry,
               **more)


class _View:
    """A device array of the library for torch; the tensor made from it keeps `owner`, whose memory it is."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False), version=2)


def _arrays(owner, handle, n_blocks, n_dof, n_qp):
    p = [C.POINTER(C.c_double)() for _ in range(5)]
    _lib.check(_lib.lib.pg_ctx_device_arrays(handle, *[C.byref(x) for x in p]))
    sizes = (4 * n_blocks, n_dof, n_dof, n_qp, n_qp)
    return [torch.as_tensor(_View(C.cast(x, C.c_void_p).value, n, owner), device=DEV) if n else None
            for x, n in zip(p, sizes)]


def _context_arrays(ctx):
    i = ctx.info
    return _arrays(ctx, ctx.handle, i["n_blocks"], i["n_dof"], i["n_cohesive_qp"])


def _cohesive(case):
    """Cohesive laws: Ortiz-Pandolfi {sigma_c, delta_c, beta, viscosity}; bilinear {sigma_c, G_c, K_p, beta}."""
    if case.get("law", COH_BILINEAR) == COH_OP:
        return dict(cohesive=True, coh_law=COH_OP, coh_params=(30.0, 0.002, 1.0, 0.5, 0.0))
    return dict(cohesive=True, coh_law=COH_BILINEAR, coh_params=(30.0, 1.0, 1.0e6, 1.0, 0.0))


def _tangent_inputs(mesh, case, seed):
    """A displacement in the softening range (strained linearly, interfaces a little open) and committed state."""
    g = torch.Generator().manual_seed(seed)
    e = mesh.export()
    xy = torch.from_numpy(e["xy"])
    nr = e["n_regular_nodes"]
    opening = 2e-3 if case["law"] == COH_OP else 2e-4
    U = torch.zeros_like(xy)
    U[:nr, 0] = 0.01 * xy[:nr, 0] + 0.002 * xy[:nr, 1] ** 2
    U[:nr, 1] = -0.003 * xy[:nr, 1] + 0.001 * xy[:nr, 0]
    U[nr:] = opening * (2.0 * torch.rand(xy[nr:].shape, generator=g, dtype=F64) - 1.0)
    isv = opening * torch.rand(mesh.info["n_cohesive_qp"], generator=g, dtype=F64)
    return U.reshape(-1), isv


def _solver_cfg(case):
    cfg = _lib.SolverCfg()
    _lib.lib.pg_solver_cfg_default(C.byref(cfg))
    cfg.precond = _lib.PG_PREC_MG
    cfg.precision = _lib.PG_PRECISION_MIXED if case.get("mixed") else _lib.PG_PRECISION_FP64
    cfg.rtol = case["rtol"]
    cfg.max_iter = 20000
    return cfg


def _batch_rves(case, seed):
    g = np.random.default_rng(case["geometry"])
    sides = [s for s in (64, 96, 128, 192, 256) if s <= case["side"]]
    return [_rve(s, s, int(g.integers(1, 65)), int(g.integers(1 << 30)), seed + k)
            for k, s in enumerate(sides[int(g.integers(len(sides)))] for _ in range(case["count"]))]


class _Batch:
    def __init__(self, meshes):
        self.meshes = meshes
        arr = (C.c_void_p * len(meshes))(*[m.handle.value for m in meshes])
        self.handle = C.c_void_p()
        _lib.check(_lib.lib.pg_batch_create(arr, len(meshes), 0, C.byref(self.handle)), "pg_batch_create")
        self.ctx = C.c_void_p(_lib.lib.pg_batch_context(self.handle))

    _destroy = _lib.lib.pg_batch_destroy

    def __del__(self):
        if self.handle:
            self._destroy(self.handle)
            self.handle = None


def _samples(rows, seed):
    """Features of the scale the predictor makes (mostly within a few units) and targets in [-1, 0]."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    X = torch.randn(rows, 16, generator=g, device=DEV)
    X[:, 12:14] = (X[:, 12:14] > 2.0).float()
    T = -torch.rand(rows, 2, generator=g, device=DEV)
    return X, T


def prepare(case, seed):
    op = case["op"]
    if op in ("mlp_forward", "mlp_train"):
        net = learned.MLP(0, seed=seed)
        X, T = _samples(case["rows"], seed)
        return dict(case=case, net=net, X=X, T=T, start=net.params())
    if op == "batch":
        b = _Batch([problem.Mesh(r) for r in _batch_rves(case, seed)])
        n_dof = sum(m.info["n_dof"] for m in b.meshes)
        n_blocks = sum(m.info["n_blocks"] for m in b.meshes)
        return dict(case=case, batch=b, U=_arrays(b, b.ctx, n_blocks, n_dof, 0)[1], cfg=_solver_cfg(case),
                    stats=_lib.SolveStats())
    coh = _cohesive(case) if op in ("tangent", "newton") else {}
    rve = _rve(case["nx"], case["ny"], case["inc"], case["geometry"], seed, strain=case.get("strain", 0.01), **coh)
    prob = (problem.ProblemNonlinearStructural if coh else problem.ProblemLinearElasticity)(rve)
    prob.init()
    K, U, F, isv_c, isv_t = _context_arrays(prob.ctx)
    state = dict(case=case, prob=prob, K=K, U=U, F=F, isv_c=isv_c, isv_t=isv_t)
    if op == "tangent":
        u, isv = _tangent_inputs(prob.mesh, case, seed)
        state["u"] = u.to(DEV)
        isv_c.copy_(isv)
    elif op == "solve" and case["mg"]:
        prob.get_solver().configure(precond=_lib.PG_PREC_MG, rtol=case["rtol"], max_iter=20000,
                                    precision=_lib.PG_PRECISION_MIXED if case["mixed"] else _lib.PG_PRECISION_FP64)
    elif op == "solve":
        prob.get_solver().cfg.rtol = case["rtol"]
    elif op == "newton":
        prob.configure(n_steps=case["steps"], precond=_lib.PG_PREC_MG, predictor=_lib.PG_PREDICT_LINEAR, rtol=1e-11,
                       stol=0.0, rtol_base=_lib.PG_RTOL_BASE_ZEROTH, lin_max_iter=1000,
                       precision=_lib.PG_PRECISION_MIXED if case["mixed"] else _lib.PG_PRECISION_FP64)
    elif op == "sensitivity":
        prob.get_solver().configure(precond=_lib.PG_PREC_MG, rtol=case["rtol"])
        prob.solve_problem()
        state["cfg"] = _solver_cfg(case)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _reset(*tensors):
    """Back to the unloaded state, written before the library's own stream reads it."""
    for t in tensors:
        t.zero_()
    torch.cuda.current_stream().synchronize()


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "assemble":
        state["prob"].get_assembler().assemble_linear()
        return state["K"]
    if op == "tangent":
        state["prob"].get_assembler().assemble_nonlinear(0.02, U_dev=state["u"].data_ptr())
        return dict(K=state["K"], F=state["F"], isv=state["isv_t"])
    if op == "solve":
        _reset(state["U"])
        state["prob"].solve_problem()
        return state["U"]
    if op == "newton":
        _reset(state["U"], state["isv_c"])
        state["prob"].solve_problem()
        return dict(U=state["U"], isv=state["isv_c"])
    if op == "batch":
        _reset(state["U"])
        b = state["batch"]
        _lib.check(_lib.lib.pg_assemble_linear(b.ctx, None), "pg_assemble_linear")
        _lib.check(_lib.lib.pg_batch_solve(b.handle, C.byref(state["cfg"]), None, C.byref(state["stats"])),
                   "pg_batch_solve")
        return state["U"]
    if op == "sensitivity":
        c11, d = C.c_double(), np.zeros(len(state["prob"].rve.inclusions))
        _lib.check(_lib.lib.pg_sensitivity_c11(state["prob"].ctx.handle, C.byref(state["cfg"]), 0.0, C.byref(c11),
                                               _lib.dptr(d), None), "pg_sensitivity_c11")
        return dict(c11=c11.value, dc11_dr=d)
    if op == "mlp_forward":
        return state["net"].forward(state["X"])
    net = state["net"]
    net.set_params(state["start"])
    loss = net.train(state["X"], state["T"], epochs=1, batch=case["batch"])
    return dict(params=net.params(), loss=loss)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(nx, ny, inc, cohesive):
    reg = (nx + 1) * (ny + 1)
    cut = int(inc * 4 * 0.3 / math.sqrt(inc) * (nx + ny + max(nx, ny)))
    enr = cut * (2 if cohesive else 1)
    return reg + enr, 7 * reg + 11 * enr, 2 * nx * ny, cut


def work(case):
    op = case["op"]
    if op in ("mlp_forward", "mlp_train"):
        flops = 2.0 * case["rows"] * (16 * 64 + 64 * 64 + 64 * 2)
        return dict(bytes=72.0 * case["rows"], flops=flops * (3 if op == "mlp_train" else 1))
    if op == "batch":
        s = [_sizes(h, h, 32, False) for h in (64, 96, 128, 192, 256) if h <= case["side"]]
        nodes, blocks, elems, cut = (case["count"] * sum(x[k] for x in s) / len(s) for k in range(4))
    else:
        nodes, blocks, elems, cut = _sizes(case["nx"], case["ny"], case["inc"], op in ("tangent", "newton"))
    mesh = 16.0 * nodes + 13.0 * elems + 64.0 * 5 * cut
    per_elem = 150.0 * elems + 4000.0 * cut
    if op == "assemble":
        return dict(bytes=mesh + 32.0 * blocks, flops=per_elem)
    if op == "tangent":
        return dict(bytes=mesh + 32.0 * blocks + 32.0 * nodes, flops=1.3 * per_elem)
    # a solve reads the matrix and the load and writes the displacements, once each
    return dict(bytes=mesh + 36.0 * blocks + 32.0 * nodes, flops=per_elem + 8.0 * blocks)


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
_TRI3 = [(1 / 3, 1 / 3, -0.28125), (0.2, 0.2, 25 / 96), (0.2, 0.6, 25 / 96), (0.6, 0.2, 25 / 96)]
# the seven-point rule at the digits in which the method's polygon rule states it
_TRI7 = [(0.33333333333333, 0.33333333333333, 0.1125)] + [
    (a, b, w) for p, q, w in ((0.47014206410511, 0.05971587178977, 0.066197076394255),
                              (0.10128650732346, 0.79742698535309, 0.062969590272415))
    for a, b in ((p, p), (p, q), (q, p))]


def _child_rule(nc):
    """(weight, shape gradients) at the quadrature points of a child element with nc nodes."""
    if nc == 3:
        return [(w, [(-1.0, -1.0), (1.0, 0.0), (0.0, 1.0)]) for _, _, w in _TRI3]
    if nc == 4:
        g, corner = 1 / math.sqrt(3.0), ((-1, -1), (1, -1), (1, 1), (-1, 1))
        return [(1.0, [(0.25 * a * (1 + b * s), 0.25 * b * (1 + a * r)) for a, b in corner])
                for s in (-g, g) for r in (-g, g)]
    # Wachspress shape functions on the regular polygon; 4 nc points of the
    # seven-point rule over the triangles around its centre
    P = [(math.cos(2 * math.pi * (k + 1) / nc), math.sin(2 * math.pi * (k + 1) / nc)) for k in range(nc)]
    out = []
    for q in range(4 * nc):
        tr, ts, tw = _TRI7[q % 7]
        a, b = P[q // 7], P[(q // 7 + 1) % nc]
        x, y = tr * a[0] + ts * b[0], tr * a[1] + ts * b[1]
        edge = []  # area towards edge (k, k+1) and its gradient
        for k in range(nc):
            (x1, y1), (x2, y2) = P[k], P[(k + 1) % nc]
            edge.append((0.5 * ((x1 - x) * (y2 - y) - (x2 - x) * (y1 - y)), 0.5 * (y1 - y2), 0.5 * (x2 - x1)))
        al = []
        for k in range(nc):
            (A0, gx0, gy0), (A1, gx1, gy1) = edge[k - 1], edge[k]
            v = 1.0 / (A0 * A1)
            al.append((v, -v * (gx0 / A0 + gx1 / A1), -v * (gy0 / A0 + gy1 / A1)))
        s = [sum(t[d] for t in al) for d in range(3)]
        out.append((tw * (a[0] * b[1] - a[1] * b[0]),
                    [((t[1] - t[0] / s[0] * s[1]) / s[0], (t[2] - t[0] / s[0] * s[2]) / s[0]) for t in al]))
    return out


def _gradients(X, dN):
    """Jacobian determinant and physical gradients of shape functions dN[k][2] on X[n, k, 2]."""
    d = torch.tensor(dN, dtype=F64, device=X.device)
    J = torch.einsum("ka,nki->nai", d, X)
    det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
    inv = torch.stack([torch.stack([J[:, 1, 1], -J[:, 0, 1]], 1), torch.stack([-J[:, 1, 0], J[:, 0, 0]], 1)], 1)
    return det, torch.einsum("nab,kb->nka", inv / det[:, None, None], d)


def _BDB(G, D):
    """Blocks B_a^T D B_b of gradients G[n, k, 2] under plane-strain moduli D[n, 3] (D11, D12, D33)."""
    xx, xy = G[:, :, None, 0] * G[:, None, :, 0], G[:, :, None, 0] * G[:, None, :, 1]
    yx, yy = G[:, :, None, 1] * G[:, None, :, 0], G[:, :, None, 1] * G[:, None, :, 1]
    a, b, c = (D[:, k, None, None] for k in range(3))
    return torch.stack([a * xx + c * yy, b * xy + c * yx, b * yx + c * xy, a * yy + c * xx], -1)


def _law(case, dt, dmax, dl):
    """Traction and tangent of the cohesive law at openings dl[n, 2] (tangential, normal), and the new delta_max."""
    p = _cohesive(case)["coh_params"]
    if case.get("law", COH_BILINEAR) == COH_OP:
        sc, dc, visc = p[0], p[1], p[3]
        beta2, dn = p[2] ** 2, dl[:, 1]
        de = torch.sqrt(dn ** 2 + beta2 * dl[:, 0] ** 2)
        ex, exm = torch.exp(1 - de / dc), torch.exp(1 - dmax / dc)
        T1 = sc * de / dc * ex + visc / sc * (de - dmax) / dt / dc
        d1 = sc / dc * (1 - de / dc) * ex + visc / sc / dt / dc
        Tm = sc * dmax / dc * exm
    else:
        sc, df, d0 = p[0], 2 * p[1] / p[0], p[0] / p[2]
        beta2, dn = p[3] ** 2, dl[:, 1].clamp(min=0)
        de = torch.sqrt(dn ** 2 + beta2 * dl[:, 0] ** 2) + 1e-300

        def env(d):
            soft = d < df
            return (torch.where(d <= d0, p[2] * d, torch.where(soft, sc * (df - d) / (df - d0), 0 * d)),
                    torch.where(d <= d0, p[2] + 0 * d, torch.where(soft, -sc / (df - d0) + 0 * d, 0 * d)))

        (T1, d1), (Tm, _) = env(de), env(dmax)
    load = de >= dmax
    T, dT = torch.where(load, T1, Tm * de / dmax), torch.where(load, d1, Tm / dmax)
    s, a = T / de, (dT * de - T) / de ** 3
    br = torch.stack([beta2 * dl[:, 0], dn], 1)
    t = s[:, None] * br
    Dc = a[:, None, None] * br[:, :, None] * br[:, None, :]
    Dc[:, 0, 0] += s * beta2
    Dc[:, 1, 1] += s
    if case.get("law", COH_BILINEAR) != COH_OP:  # compression: the penalty stiffness, uncoupled
        c = dl[:, 1] < 0
        t[c, 1] = p[2] * dl[c, 1]
        Dc[c, 0, 1] = Dc[c, 1, 0] = 0.0
        Dc[c, 1, 1] = p[2]
    return t, Dc, torch.where(load, de, dmax)


def _exact_system(rve, mesh, u=None, isv=None, case=None, dt=1.0):
    """K in the mesh's block pattern, and with u the internal force and the trial state, summed in plain torch
    from the mesh's nodes, connectivity and cut templates."""
    e = mesh.export()
    to = lambda v: torch.as_tensor(np.ascontiguousarray(v)).to(DEV)  # noqa: E731
    xy, conn, n = to(e["xy"]), to(e["conn"]).long(), e["xy"].shape[0]
    rp, col = to(e["row_ptr"]).long(), to(e["col"]).long()
    keys = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1]) * n + col
    K = torch.zeros(keys.numel(), 4, dtype=F64, device=DEV)
    F = torch.zeros(n, 2, dtype=F64, device=DEV)
    isv_t = None if isv is None else isv.clone()
    D = torch.tensor([[E / ((1 + v) * (1 - 2 * v)) * f for f in (1 - v, v, (1 - 2 * v) / 2)]
                      for E, v in rve.materials], dtype=F64, device=DEV)

    def add(nodes, blocks):
        at = torch.searchsorted(keys, (nodes[:, :, None] * n + nodes[:, None, :]).reshape(-1))
        K.index_add_(0, at, blocks.reshape(-1, 4))
        if u is not None:
            k = blocks.reshape(*blocks.shape[:3], 2, 2)
            F.index_add_(0, nodes.reshape(-1), torch.einsum("nabij,nbj->nai", k, u[nodes]).reshape(-1, 2))

    whole = to(e["elem_cut"]) < 0
    nodes = conn[whole]
    det, G = _gradients(xy[nodes], [(-1.0, -1.0), (1.0, 0.0), (0.0, 1.0)])
    add(nodes, 0.5 * det[:, None, None, None] * _BDB(G, D[to(e["elem_mat"]).long()[whole]]))
    tmpl, cut_elem = to(e["cut_tmpl"]), to(e["cut_elem"]).long()
    enr, chm, qp0 = to(e["cut_enr"]).long(), to(e["cut_child_mat"]).long(), to(e["cut_coh_qp0"]).long()
    for t, row in enumerate(problem.template_table().tolist()):
        sel = torch.nonzero(tmpl == t).reshape(-1)
        if not sel.numel():
            continue
        n_enr, n_child, n_coh = row[1:4]
        child_n, child_nodes, coh_nodes = row[16:20], row[24:48], row[48:60]
        nl = 3 + n_enr
        nodes = torch.cat([conn[cut_elem[sel]], enr[sel, :n_enr]], 1)
        X = xy[nodes]
        _, parent = _gradients(X[:, :3], [(-1.0, -1.0), (1.0, 0.0), (0.0, 1.0)])
        blocks = torch.zeros(sel.numel(), nl, nl, 4, dtype=F64, device=DEV)
        for c in range(n_child):
            loc = child_nodes[6 * c:6 * c + child_n[c]]
            Dc = D[chm[sel, c]]
            for w, dN in _child_rule(child_n[c]):
                det, g = _gradients(X[:, loc], dN)
                G = torch.zeros(sel.numel(), nl, 2, dtype=F64, device=DEV)
                G[:, :3] = parent
                for k, a in enumerate(loc):
                    if a >= 3:
                        G[:, a] = g[:, k]
                live = (det * w != 0)[:, None, None, None]  # a collapsed child adds nothing
                blocks += torch.where(live, (det * w)[:, None, None, None] * _BDB(G, Dc), torch.zeros_like(blocks))
        add(nodes, blocks)
        if u is None or not n_coh:
            continue
        for c in range(n_coh):
            loc = coh_nodes[4 * c:4 * c + 4]
            N, Y = nodes[:, loc], X[:, loc]
            tang = 0.5 * (Y[:, 1] - Y[:, 0])
            dA = tang.norm(dim=1)
            R = torch.stack([tang, torch.stack([-tang[:, 1], tang[:, 0]], 1)], 1) / dA[:, None, None]
            live = dA != 0
            for q, xi in enumerate((-1 / math.sqrt(3.0), 1 / math.sqrt(3.0))):
                B = torch.tensor([-(1 - xi) / 2, -(1 + xi) / 2, (1 - xi) / 2, (1 + xi) / 2], dtype=F64, device=DEV)
                dl = torch.einsum("nij,k,nkj->ni", R, B, u[N])
                at = qp0[sel] + 2 * c + q
                tr, T, isv_t[at] = _law(case, dt, isv[at], dl)
                T = torch.einsum("nai,nab,nbj->nij", R, T, R)
                blk = torch.einsum("n,k,l,nij->nklij", dA, B, B, T).reshape(-1, 4, 4, 4)
                where = torch.searchsorted(keys, (N[:, :, None] * n + N[:, None, :]).reshape(-1))
                blk = torch.where(live[:, None, None, None], blk, torch.zeros_like(blk))
                K.index_add_(0, where, blk.reshape(-1, 4))
                f = torch.einsum("n,k,nai,na->nki", dA, B, R, tr)
                F.index_add_(0, N.reshape(-1), torch.where(live[:, None, None], f, torch.zeros_like(f)).reshape(-1, 2))
    return dict(K=K.reshape(-1), F=F.reshape(-1), isv=isv_t, row_ptr=rp, col=col,
                fixed=to(e["fixed"]), ubar=to(e["ubar"]))


def _exact_solution(system):
    """Displacements under the prescribed values: block-Jacobi CG to rounding."""
    rp, col, fixed = system["row_ptr"], system["col"], system["fixed"]
    K = system["K"].reshape(-1, 2, 2)
    n = rp.numel() - 1
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    width = rp[1:] - rp[:-1]
    # block CSR to scalar CSR: each row of a node holds its blocks' first or second rows
    crow = torch.zeros(2 * n + 1, dtype=torch.long, device=DEV)
    crow[1:] = torch.cumsum(torch.stack([2 * width, 2 * width], 1).reshape(-1), 0)
    k = torch.arange(col.numel(), device=DEV) - rp[rows]
    ccol = torch.empty(int(crow[-1]), dtype=torch.long, device=DEV)
    val = torch.empty(int(crow[-1]), dtype=F64, device=DEV)
    for d in range(2):
        for f in range(2):
            at = crow[2 * rows + d] + 2 * k + f
            ccol[at] = 2 * col + f
            val[at] = K[:, d, f]
    A = torch.sparse_csr_tensor(crow, ccol, val, size=(2 * n, 2 * n))
    free = (~fixed).double()
    up = system["ubar"] * (1 - free)
    M = K[rows == col] * free.reshape(n, 2, 1) * free.reshape(n, 1, 2) + torch.diag_embed((1 - free).reshape(n, 2))
    M = torch.linalg.inv(M)
    pre = lambda v: torch.einsum("nij,nj->ni", M, v.reshape(n, 2)).reshape(-1) * free  # noqa: E731
    x, r = torch.zeros_like(up), -(A @ up) * free
    z = pre(r)
    p, rz, first = z, torch.dot(r, z), float(torch.dot(r, r))
    for it in range(20000):
        q = (A @ p) * free
        a = rz / torch.dot(p, q)
        x, r = x + a * p, r - a * q
        if it % 50 == 0 and float(torch.dot(r, r)) <= 1e-29 * first:
            break
        z = pre(r)
        rz, old = torch.dot(r, z), rz
        p = z + rz / old * p
    return x + up


def exact(case, seed):
    op = case["op"]
    if op == "mlp_forward":
        return _network(_split(torch.from_numpy(learned.MLP(0, seed=seed).params()).to(DEV).double()),
                        _samples(case["rows"], seed)[0].double())
    if op == "mlp_train":
        return _exact_training(case, seed)
    if op == "batch":
        return torch.cat([_exact_solution(_exact_system(r, problem.Mesh(r))) for r in _batch_rves(case, seed)])
    if op in ("newton", "sensitivity"):
        return None  # a whole load path, an adjoint with element derivatives: no plain form within seconds
    if op == "solve" and case["nx"] * case["ny"] > 300000:
        return None  # the plain iteration takes longer than is worth waiting for
    coh = _cohesive(case) if op == "tangent" else {}
    rve = _rve(case["nx"], case["ny"], case["inc"], case["geometry"], seed, **coh)
    mesh = problem.Mesh(rve)
    if op == "tangent":
        u, isv = _tangent_inputs(mesh, case, seed)
        s = _exact_system(rve, mesh, u.reshape(-1, 2).to(DEV), isv.to(DEV), case, 0.02)
        return dict(K=s["K"], F=s["F"], isv=s["isv"])
    s = _exact_system(rve, mesh)
    return s["K"] if op == "assemble" else _exact_solution(s)


def _split(v):
    out, at = [], 0
    for shape in ((64, 16), (64,), (64, 64), (64,), (16, 64), (16,)):
        size = math.prod(shape)
        out.append(v[at:at + size].reshape(shape))
        at += size
    return out


def _network(p, X):
    W1, b1, W2, b2, W3, b3 = p
    return (torch.relu(torch.relu(X @ W1.T + b1) @ W2.T + b2) @ W3.T + b3)[:, :2]


def _exact_training(case, seed):
    X, T = (v.double() for v in _samples(case["rows"], seed))
    v = torch.from_numpy(learned.MLP(0, seed=seed).params()).to(DEV).double().requires_grad_()
    m1, m2, losses = torch.zeros_like(v), torch.zeros_like(v), []
    for k, at in enumerate(range(0, case["rows"], case["batch"])):
        x, t = X[at:at + case["batch"]], T[at:at + case["batch"]]
        loss = (_network(_split(v), x) - t).square().sum() / x.shape[0]
        g, = torch.autograd.grad(loss, v)
        with torch.no_grad():
            m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
            v -= 2e-3 * (m1 / (1 - 0.9 ** (k + 1))) / (torch.sqrt(m2 / (1 - 0.999 ** (k + 1))) + 1e-8)
        losses.append(float(loss.detach()))
    return dict(params=v.detach(), loss=np.array([np.mean(losses)]))
