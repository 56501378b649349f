// Many independent linear-elastic RVEs of uneven size assembled and solved
// together (sm_100a).
//
// The reference solves one RVE per run (Problem::solve_problem,
// src/Problem.cpp:400-418); a batch here is the block-diagonal union of the
// RVEs' IGFEM systems.  The meshes are concatenated node by node (each RVE's
// regular then enrichment nodes), so one launch of each assembly kernel
// covers every RVE, and the solve is CG with per-RVE scalars: every RVE has
// its own step lengths, its own residual target (rtol times its own right-
// hand side) and stops on its own, while the kernels keep running over the
// whole batch until the last RVE converges.  The preconditioner is either
// block Jacobi or one multigrid V-cycle of every RVE's own grid hierarchy
// (pg_mg.cu, whose kernels cover all the RVEs of a context).  The CG
// iterations of a whole batch run as CUDA graphs.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <sys/mman.h>
#include <vector>

#include "pg_solve_kernels.cuh"
#include "pigfem_b200.h"

namespace pgb {

namespace {

inline int nb(long long n, int t = kThreads) { return (int)((n + t - 1) / t); }

// z = M^-1 r (block Jacobi), whole batch
__global__ void k_b_jacobi(int n, const double* __restrict__ minv, const double* __restrict__ r, double* __restrict__ z,
                           const int* done) {
    if (done && done[0]) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* m = minv + 4 * (size_t)i;
    const double r0 = r[2 * i], r1 = r[2 * i + 1];
    z[2 * i] = m[0] * r0 + m[1] * r1;
    z[2 * i + 1] = m[2] * r0 + m[3] * r1;
}

// ---------------------------------------------------------------------------
// Per-RVE CG.  Scalars per RVE (8 doubles): 0 p.q, 1 r.z, 2 new r.z, 3 r.r,
// 4 tol^2, 5 b.b, 6 true r.r; flags per RVE (4 ints): 0 done, 1 breakdown,
// 2 iterations.  g[0]: RVEs done, g[1]: all done.
// ---------------------------------------------------------------------------
// Segmented sum: lanes of a warp that share one RVE reduce by shuffles; a
// warp that straddles two RVEs adds lane by lane.
__device__ __forceinline__ void seg_add(double v, int rve, double* acc, int stride, int slot) {
    const unsigned full = 0xffffffffu;
    const int r0 = __shfl_sync(full, rve, 0);
    if (__all_sync(full, rve == r0)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(full, v, o);
        if ((threadIdx.x & 31) == 0 && rve >= 0) atomicAdd(&acc[(size_t)rve * stride + slot], v);
    } else if (rve >= 0 && v != 0.0) {
        atomicAdd(&acc[(size_t)rve * stride + slot], v);
    }
}

__global__ void __launch_bounds__(kThreads) k_bcg_start(int nd, const int* __restrict__ node_rve,
                                                        const uint8_t* __restrict__ fixed, const double* __restrict__ b,
                                                        double* __restrict__ r, double* __restrict__ x, double* sc) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    double v = 0.0;
    int rve = -1;
    if (i < nd) {
        v = fixed[i] ? 0.0 : b[i];
        r[i] = v;
        x[i] = 0.0;
        rve = node_rve[i >> 1];
    }
    seg_add(v * v, rve, sc, 8, 3);
}

__global__ void k_bcg_tol(int nr, double* sc, int* fl, int* g, double rtol2) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    double* s = sc + 8 * r;
    s[5] = s[3];
    s[4] = rtol2 * s[3];
    if (s[3] == 0.0) {
        fl[4 * r] = 1;
        atomicAdd(&g[0], 1);
    }
}

__global__ void k_bcg_alldone(int nr, int* g) {
    if (g[0] >= nr) g[1] = 1;
}

__global__ void k_bcg_s1(int nr, double* sc, const int* fl, const int* g) {
    if (g[1]) return;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr || fl[4 * r]) return;
    double* s = sc + 8 * r;
    s[1] = s[2];
    s[0] = 0.0;
    s[3] = 0.0;
}

__global__ void __launch_bounds__(kThreads) k_bcg_spmv(int n, const int* __restrict__ node_rve,
                                                       const int* __restrict__ row_ptr, const int* __restrict__ col,
                                                       const double* __restrict__ K, const double* __restrict__ p,
                                                       const uint8_t* __restrict__ fixed, double* __restrict__ q,
                                                       double* sc, const int* g) {
    if (g[1]) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    double part = 0.0;
    int rve = -1;
    if (i < n) {
        double y0, y1;
        bsr_row<double, double>(i, row_ptr, col, K, p, y0, y1);
        if (fixed[2 * i]) y0 = 0.0;
        if (fixed[2 * i + 1]) y1 = 0.0;
        q[2 * i] = y0;
        q[2 * i + 1] = y1;
        part = p[2 * i] * y0 + p[2 * i + 1] * y1;
        rve = node_rve[i];
    }
    seg_add(part, rve, sc, 8, 0);
}

__global__ void __launch_bounds__(kThreads) k_bcg_update(int nd, const int* __restrict__ node_rve,
                                                         double* __restrict__ x, double* __restrict__ r,
                                                         const double* __restrict__ p, const double* __restrict__ q,
                                                         double* sc, int* fl, const int* g) {
    if (g[1]) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    double part = 0.0;
    int rve = -1;
    if (i < nd) {
        rve = node_rve[i >> 1];
        const double* s = sc + 8 * rve;
        if (!fl[4 * rve]) {
            const double pq = s[0];
            if (pq > 0.0) {
                const double alpha = s[1] / pq;
                x[i] += alpha * p[i];
                const double ri = r[i] - alpha * q[i];
                r[i] = ri;
                part = ri * ri;
            } else {
                fl[4 * rve + 1] = 1;
            }
        }
    }
    seg_add(part, rve, sc, 8, 3);
}

__global__ void k_bcg_s2(int nr, double* sc, int* fl, int* g) {
    if (g[1]) return;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr || fl[4 * r]) return;
    double* s = sc + 8 * r;
    fl[4 * r + 2] += 1;
    if (fl[4 * r + 1] || s[3] <= s[4]) {
        fl[4 * r] = 1;
        atomicAdd(&g[0], 1);
    }
    s[2] = 0.0;
}

__global__ void __launch_bounds__(kThreads) k_bcg_dot(int nd, const int* __restrict__ node_rve, const double* __restrict__ a,
                                                      const double* __restrict__ b, double* sc, int slot, const int* g) {
    if (g && g[1]) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    double v = 0.0;
    int rve = -1;
    if (i < nd) {
        v = a[i] * b[i];
        rve = node_rve[i >> 1];
    }
    seg_add(v, rve, sc, 8, slot);
}

__global__ void __launch_bounds__(kThreads) k_bcg_pupdate(int nd, const int* __restrict__ node_rve,
                                                          const double* __restrict__ z, double* __restrict__ p,
                                                          const double* sc, const int* fl, const int* g) {
    if (g[1]) return;
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= nd) return;
    const int rve = node_rve[i >> 1];
    if (fl[4 * rve]) return;
    const double* s = sc + 8 * rve;
    p[i] = z[i] + (s[2] / s[1]) * p[i];
}

template <typename T>
int b_alloc(std::vector<void*>& owned, T** p, size_t n) {
    *p = nullptr;
    PG_CUDA(cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(T)));
    PG_CUDA(fill_sync(*p, 0, std::max<size_t>(n, 1) * sizeof(T)));
    owned.push_back((void*)*p);
    return PG_OK;
}

template <typename T>
int b_upload(std::vector<void*>& owned, T** p, const std::vector<T>& v) {
    int rc = b_alloc(owned, p, v.size());
    if (rc) return rc;
    if (!v.empty()) PG_CUDA(h2d_sync(*p, v.data(), v.size() * sizeof(T)));
    return PG_OK;
}

}  // namespace
}  // namespace pgb

struct pg_batch {
    int n_rve = 0;
    // host seconds of the set-up: mesh copies, merge, context (uploads, grid
    // tiles, cut tables, fold order), multigrid hierarchy
    double setup_s[7] = {0, 0, 0, 0, 0, 0, 0};
    std::vector<std::pair<int, int>> grid;  // background grid (nx, ny) of each RVE
    std::vector<int> noff;              // first node of each RVE (+ total)
    std::vector<int> eoff;              // first element of each RVE (+ total)
    pg_ctx ctx;                         // the merged system
    std::vector<int> depth;             // multigrid depth per RVE
    int* node_rve0 = nullptr;           // batch nodes -> RVE
    // per-RVE CG
    double* sc = nullptr;
    int* fl = nullptr;
    int* g = nullptr;
    std::vector<void*> owned;
};

namespace pgb {
namespace {

// Concatenates the RVE meshes into one block-diagonal mesh: every array's
// place per RVE first (prefix sums of the sizes), then the RVEs copied and
// renumbered in parallel, each into its own range.
void merge_meshes(const pg_mesh* const* ms, int R, HostMesh& out, std::vector<int>& noff, std::vector<int>& eoff) {
    out = HostMesh();
    auto M = [&](int r) -> const HostMesh& { return ms[r]->m; };
    noff.assign(R + 1, 0);
    eoff.assign(R + 1, 0);
    std::vector<int> moff(R + 1, 0), coff(R + 1, 0), boff(R + 1, 0), qoff(R + 1, 0), koff(R + 1, 0);
    for (int r = 0; r < R; ++r) {
        noff[r + 1] = noff[r] + M(r).n_nodes();
        eoff[r + 1] = eoff[r] + M(r).n_elem;
        moff[r + 1] = moff[r] + (int)M(r).spec.materials.size();
        coff[r + 1] = coff[r] + M(r).n_cut;
        boff[r + 1] = boff[r] + M(r).n_blocks();
        qoff[r + 1] = qoff[r] + M(r).n_coh_qp;
        koff[r + 1] = koff[r] + (int)M(r).ne_list.size();
    }
    // the place of each RVE's part of one array, and the array sized to all
    // (its pages backed by huge pages where the host allows it: sizing a
    // multi-GB array otherwise costs a page fault per 4 KB)
    auto place = [&](auto field, auto& dst) {
        std::vector<size_t> o(R + 1, 0);
        for (int r = 0; r < R; ++r) o[r + 1] = o[r] + (M(r).*field).size();
        dst.reserve(o[R]);
        const size_t bytes = o[R] * sizeof(dst[0]);
        if (bytes >= (8u << 20)) {
            const uintptr_t a = (reinterpret_cast<uintptr_t>(dst.data()) + 4095) & ~uintptr_t(4095);
            const uintptr_t e = reinterpret_cast<uintptr_t>(dst.data()) + bytes;
            if (e > a) madvise(reinterpret_cast<void*>(a), e - a, MADV_HUGEPAGE);
        }
        dst.resize(o[R]);
        return o;
    };
    const auto o_x = place(&HostMesh::x, out.x);
    place(&HostMesh::y, out.y);
    const auto o_conn = place(&HostMesh::conn, out.conn);
    const auto o_emat = place(&HostMesh::elem_mat, out.elem_mat);
    place(&HostMesh::elem_cut, out.elem_cut);
    const auto o_cut = place(&HostMesh::cut_elem, out.cut_elem);
    place(&HostMesh::cut_tmpl, out.cut_tmpl);
    const auto o_cenr = place(&HostMesh::cut_enr, out.cut_enr);
    const auto o_cchm = place(&HostMesh::cut_child_mat, out.cut_child_mat);
    const auto o_ccoh = place(&HostMesh::cut_coh_mat, out.cut_coh_mat);
    place(&HostMesh::cut_coh_qp0, out.cut_coh_qp0);
    const auto o_fix = place(&HostMesh::fixed, out.fixed);
    place(&HostMesh::ubar, out.ubar);
    const auto o_col = place(&HostMesh::col, out.col);
    const auto o_diag = place(&HostMesh::diag_slot, out.diag_slot);
    const auto o_nel = place(&HostMesh::ne_list, out.ne_list);
    const auto o_slot = place(&HostMesh::cut_slot, out.cut_slot);
    out.row_ptr.assign((size_t)noff[R] + 1, 0);
    out.ne_ptr.assign((size_t)noff[R] + 1, 0);
    parallel_for(R, 1, [&](long long rr) {
        const int r = (int)rr;
        const HostMesh& m = M(r);
        const int no = noff[r], eo = eoff[r], mo = moff[r], co = coff[r], bo = boff[r], qo = qoff[r], ko = koff[r];
        std::copy(m.x.begin(), m.x.end(), out.x.begin() + o_x[r]);
        std::copy(m.y.begin(), m.y.end(), out.y.begin() + o_x[r]);
        for (size_t i = 0; i < m.conn.size(); ++i) out.conn[o_conn[r] + i] = m.conn[i] + no;
        for (size_t i = 0; i < m.elem_mat.size(); ++i) {
            out.elem_mat[o_emat[r] + i] = m.elem_mat[i] + mo;
            out.elem_cut[o_emat[r] + i] = m.elem_cut[i] >= 0 ? m.elem_cut[i] + co : -1;
        }
        for (size_t i = 0; i < m.cut_elem.size(); ++i) {
            out.cut_elem[o_cut[r] + i] = m.cut_elem[i] + eo;
            out.cut_tmpl[o_cut[r] + i] = m.cut_tmpl[i];
            out.cut_coh_qp0[o_cut[r] + i] = m.cut_coh_qp0[i] + qo;
        }
        for (size_t i = 0; i < m.cut_enr.size(); ++i) out.cut_enr[o_cenr[r] + i] = m.cut_enr[i] >= 0 ? m.cut_enr[i] + no : -1;
        for (size_t i = 0; i < m.cut_child_mat.size(); ++i)
            out.cut_child_mat[o_cchm[r] + i] = m.cut_child_mat[i] >= 0 ? m.cut_child_mat[i] + mo : -1;
        std::copy(m.cut_coh_mat.begin(), m.cut_coh_mat.end(), out.cut_coh_mat.begin() + o_ccoh[r]);
        std::copy(m.fixed.begin(), m.fixed.end(), out.fixed.begin() + o_fix[r]);
        std::copy(m.ubar.begin(), m.ubar.end(), out.ubar.begin() + o_fix[r]);
        for (size_t i = 1; i < m.row_ptr.size(); ++i) out.row_ptr[no + i] = m.row_ptr[i] + bo;
        for (size_t i = 0; i < m.col.size(); ++i) out.col[o_col[r] + i] = m.col[i] + no;
        for (size_t i = 0; i < m.diag_slot.size(); ++i) out.diag_slot[o_diag[r] + i] = m.diag_slot[i] + bo;
        for (size_t i = 1; i < m.ne_ptr.size(); ++i) out.ne_ptr[no + i] = m.ne_ptr[i] + ko;
        for (size_t i = 0; i < m.ne_list.size(); ++i) {
            const int v = m.ne_list[i];
            out.ne_list[o_nel[r] + i] = (((v >> 2) + eo) << 2) | (v & 3);
        }
        for (size_t i = 0; i < m.cut_slot.size(); ++i) out.cut_slot[o_slot[r] + i] = m.cut_slot[i] >= 0 ? m.cut_slot[i] + bo : -1;
    });
    out.spec = M(0).spec;
    out.spec.materials.clear();
    out.spec.inclusions.clear();
    out.spec.nx = out.spec.ny = 0;
    out.n_reg = noff[R];  // every node counts as "regular" for the batch-level views
    out.n_enr = 0;
    out.n_elem = eoff[R];
    out.n_cut = coff[R];
    out.n_coh_qp = qoff[R];
    for (int r = 0; r < R; ++r) {
        const HostMesh& m = M(r);
        out.spec.materials.insert(out.spec.materials.end(), m.spec.materials.begin(), m.spec.materials.end());
        out.n_free += m.n_free;
        for (const auto& gb : m.grids)
            out.grids.push_back({gb.nx, gb.ny, gb.node_off + noff[r], gb.elem_off + eoff[r], gb.n_reg});
    }
}

// The RVEs' multigrid hierarchies, the node map and the CG scalars (once per batch).
int batch_build(pg_batch& B) {
    Ctx& c = B.ctx.c;
    const int R = B.n_rve;
    auto& own = B.owned;
    int rc = mg_build(c);
    if (rc) return rc;
    mg_depths(c, B.depth);
    std::vector<int> nr0(B.noff[R]);
    for (int r = 0; r < R; ++r)
        for (int i = B.noff[r]; i < B.noff[r + 1]; ++i) nr0[i] = r;
    if ((rc = b_upload(own, &B.node_rve0, nr0))) return rc;
    if ((rc = b_alloc(own, &B.sc, 8 * (size_t)R)) || (rc = b_alloc(own, &B.fl, 4 * (size_t)R)) || (rc = b_alloc(own, &B.g, 8)))
        return rc;
    PG_CUDA(cudaStreamSynchronize(c.stream));
    return PG_OK;
}

// Block-Jacobi (or plain) CG on every RVE, in graphs of `chunk` iterations; the host copies of the scalars and flags.
int batch_cg(pg_batch& B, const pg_solver_cfg& cfg, std::vector<double>& hs, std::vector<int>& hf, cudaStream_t s) {
    Ctx& c = B.ctx.c;
    const int R = B.n_rve, n = c.n_nodes, nd = c.n_dof;
    k_prec_setup<double><<<nb(n), kThreads, 0, s>>>(n, c.diag, c.K, c.fixed, cfg.precond == PG_PREC_BLOCK_JACOBI,
                                                    cfg.precond == PG_PREC_NONE, c.minv);
    cudaMemsetAsync(B.fl, 0, 4 * (size_t)R * sizeof(int), s);
    cudaMemsetAsync(B.g, 0, 8 * sizeof(int), s);
    k_bcg_start<<<nb(nd), kThreads, 0, s>>>(nd, B.node_rve0, c.fixed, c.b, c.r, c.dx, B.sc);
    k_bcg_tol<<<nb(R, 128), 128, 0, s>>>(R, B.sc, B.fl, B.g, cfg.rtol * cfg.rtol);
    k_bcg_alldone<<<1, 1, 0, s>>>(R, B.g);
    k_b_jacobi<<<nb(n), kThreads, 0, s>>>(n, c.minv, c.r, c.z, nullptr);
    cudaMemcpyAsync(c.p, c.z, (size_t)nd * sizeof(double), cudaMemcpyDeviceToDevice, s);
    k_bcg_dot<<<nb(nd), kThreads, 0, s>>>(nd, B.node_rve0, c.r, c.z, B.sc, 2, nullptr);
    const int chunk = cfg.check_every > 1 ? cfg.check_every : 32;
    cudaGraph_t graph;
    PG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    for (int it = 0; it < chunk; ++it) {
        k_bcg_s1<<<nb(R, 128), 128, 0, s>>>(R, B.sc, B.fl, B.g);
        k_bcg_spmv<<<nb(n), kThreads, 0, s>>>(n, B.node_rve0, c.row_ptr, c.col, c.K, c.p, c.fixed, c.q, B.sc, B.g);
        k_bcg_update<<<nb(nd), kThreads, 0, s>>>(nd, B.node_rve0, c.dx, c.r, c.p, c.q, B.sc, B.fl, B.g);
        k_bcg_s2<<<nb(R, 128), 128, 0, s>>>(R, B.sc, B.fl, B.g);
        k_bcg_alldone<<<1, 1, 0, s>>>(R, B.g);
        k_b_jacobi<<<nb(n), kThreads, 0, s>>>(n, c.minv, c.r, c.z, B.g + 1);
        k_bcg_dot<<<nb(nd), kThreads, 0, s>>>(nd, B.node_rve0, c.r, c.z, B.sc, 2, B.g);
        k_bcg_pupdate<<<nb(nd), kThreads, 0, s>>>(nd, B.node_rve0, c.z, c.p, B.sc, B.fl, B.g);
    }
    PG_CUDA(cudaStreamEndCapture(s, &graph));
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return cuda_fail(ie, "pg_batch_solve graph");
    int hg[8] = {};
    int launched = 0;
    while (true) {
        cudaGraphLaunch(exec, s);
        launched += chunk;
        cudaMemcpyAsync(hg, B.g, sizeof hg, cudaMemcpyDeviceToHost, s);
        const cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            cudaGraphExecDestroy(exec);
            return cuda_fail(e, "pg_batch_solve");
        }
        if (hg[1] || launched >= cfg.max_iter) break;
    }
    cudaGraphExecDestroy(exec);
    cudaMemcpyAsync(hs.data(), B.sc, hs.size() * sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(hf.data(), B.fl, hf.size() * sizeof(int), cudaMemcpyDeviceToHost, s);
    PG_CUDA(cudaStreamSynchronize(s));
    return PG_OK;
}

}  // namespace
}  // namespace pgb

using namespace pgb;

extern "C" {

int pg_batch_create(const pg_mesh* const* meshes, int32_t n_rve, int32_t device, pg_batch** out) {
    if (!meshes || !out || n_rve <= 0) { set_error("pg_batch_create: invalid argument"); return PG_ERR_ARG; }
    *out = nullptr;
    for (int r = 0; r < n_rve; ++r) {
        if (!meshes[r]) { set_error("pg_batch_create: null mesh"); return PG_ERR_ARG; }
        if (meshes[r]->m.spec.cohesive) {
            set_error("pg_batch_create: batches hold linear-elastic RVEs (no cohesive interfaces)");
            return PG_ERR_ARG;
        }
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        set_error("pg_batch_create: no CUDA device (this library has no CPU fallback)");
        return PG_ERR_CUDA;
    }
    if (device < 0 || device >= ndev) { set_error("pg_batch_create: invalid device"); return PG_ERR_ARG; }
    pg_batch* B = new (std::nothrow) pg_batch;
    if (!B) { set_error("pg_batch_create: out of host memory"); return PG_ERR_ARG; }
    B->n_rve = n_rve;
    auto now = [] { return std::chrono::steady_clock::now(); };
    auto secs = [](auto a, auto b) { return std::chrono::duration<double>(b - a).count(); };
    auto t0 = now();
    for (int r = 0; r < n_rve; ++r) B->grid.push_back({meshes[r]->m.spec.nx, meshes[r]->m.spec.ny});
    auto t1 = now();
    HostMesh merged;
    merge_meshes(meshes, n_rve, merged, B->noff, B->eoff);
    auto t2 = now();
    int rc = ctx_create(std::move(merged), device, B->ctx.c);
    auto t3 = now();
    if (rc == PG_OK) rc = batch_build(*B);
    B->setup_s[0] = secs(t0, t1);
    B->setup_s[1] = secs(t1, t2);
    for (int k = 0; k < 4; ++k) B->setup_s[2 + k] = B->ctx.c.setup_s[k];
    B->setup_s[6] = secs(t3, now());
    if (rc != PG_OK) {
        pg_batch_destroy(B);
        return rc;
    }
    *out = B;
    return PG_OK;
}

void pg_batch_destroy(pg_batch* B) {
    if (!B) return;
    cudaSetDevice(B->ctx.c.device);
    for (void* p : B->owned) cudaFree(p);
    free_ctx(B->ctx.c);
    delete B;
}

pg_ctx* pg_batch_context(pg_batch* B) { return B ? &B->ctx : nullptr; }

int pg_batch_setup_times(const pg_batch* B, double* seconds) {
    if (!B || !seconds) { set_error("pg_batch_setup_times: null argument"); return PG_ERR_ARG; }
    for (int k = 0; k < 7; ++k) seconds[k] = B->setup_s[k];
    return PG_OK;
}

int pg_batch_info(const pg_batch* B, int32_t* node_offset, int32_t* element_offset, int32_t* depth) {
    if (!B) { set_error("pg_batch_info: null batch"); return PG_ERR_ARG; }
    for (int r = 0; r <= B->n_rve; ++r) {
        if (node_offset) node_offset[r] = B->noff[r];
        if (element_offset) element_offset[r] = B->eoff[r];
    }
    if (depth)
        for (int r = 0; r < B->n_rve; ++r) depth[r] = B->depth[r];
    return PG_OK;
}

int pg_batch_solve(pg_batch* B, const pg_solver_cfg* cfg, pg_solve_stats* per_rve, pg_solve_stats* total) {
    if (!B || !cfg) { set_error("pg_batch_solve: invalid argument"); return PG_ERR_ARG; }
    Ctx& c = B->ctx.c;
    cudaSetDevice(c.device);
    if (cfg->krylov != PG_KRYLOV_CG) { set_error("pg_batch_solve: batches are solved by CG"); return PG_ERR_ARG; }
    cudaStream_t s = c.stream;
    const int R = B->n_rve, nd = c.n_dof;
    cudaEventRecord(c.ev0, s);
    if (!c.assembled) {
        int rc = launch_assemble(c, c.U, 0.0, false, true, s);
        if (rc) return rc;
        c.assembled = true;
    }
    // b = mask(-K U_p) with every RVE's prescribed values at load factor 1
    set_prescribed(c, 1.0, s);
    residual_into(c, s, c.U, nullptr, c.b);
    cudaMemsetAsync(B->sc, 0, 8 * (size_t)R * sizeof(double), s);
    std::vector<double> hs(8 * (size_t)R);
    std::vector<int> hf(4 * (size_t)R);
    if (cfg->precond == PG_PREC_MG) {
        MgCgResult res;
        const int rc = mg_cg(c, *cfg, res, s);
        if (rc == PG_ERR_BREAKDOWN) set_error("pg_batch_solve: singular coarsest operator in one RVE");
        if (rc != PG_OK) return rc;
        std::copy(res.scalars, res.scalars + hs.size(), hs.begin());
        std::copy(res.flags, res.flags + hf.size(), hf.begin());
    } else {
        const int rc = batch_cg(*B, *cfg, hs, hf, s);
        if (rc != PG_OK) return rc;
    }
    // true residual per RVE
    residual_into(c, s, c.dx, c.b, c.r);
    cudaMemsetAsync(B->sc, 0, 8 * (size_t)R * sizeof(double), s);
    k_bcg_dot<<<nb(nd), kThreads, 0, s>>>(nd, B->node_rve0, c.r, c.r, B->sc, 6, nullptr);
    k_axpy_free<double><<<nb(nd), kThreads, 0, s>>>(nd, c.fixed, c.U, c.dx, 1.0);
    cudaEventRecord(c.ev1, s);
    std::vector<double> true_rr(8 * (size_t)R);
    cudaMemcpyAsync(true_rr.data(), B->sc, true_rr.size() * sizeof(double), cudaMemcpyDeviceToHost, s);
    PG_CUDA(cudaStreamSynchronize(s));
    for (int r = 0; r < R; ++r) hs[8 * r + 6] = true_rr[8 * r + 6];
    float ms = 0.f;
    cudaEventElapsedTime(&ms, c.ev0, c.ev1);
    int worst = PG_OK, max_it = 0, n_bad = 0;
    double worst_rel = 0.0;
    for (int r = 0; r < R; ++r) {
        pg_solve_stats st{};
        st.iterations = hf[4 * r + 2];
        const double bb = hs[8 * r + 5];
        st.rel_residual = bb > 0.0 ? std::sqrt(hs[8 * r + 6] / bb) : 0.0;
        st.seconds = ms * 1e-3;
        if (hf[4 * r + 1]) st.status = PG_ERR_BREAKDOWN;
        else if (!(hs[8 * r + 6] <= 4.0 * cfg->rtol * cfg->rtol * bb)) st.status = PG_ERR_NOT_CONVERGED;
        else st.status = PG_OK;
        if (st.status != PG_OK) {
            ++n_bad;
            worst = st.status;
        }
        max_it = std::max(max_it, st.iterations);
        worst_rel = std::max(worst_rel, st.rel_residual);
        if (per_rve) per_rve[r] = st;
    }
    if (total) {
        total->iterations = max_it;
        total->refinements = 0;
        total->rel_residual = worst_rel;
        total->seconds = ms * 1e-3;
        total->newton_iterations = 0;
        total->status = worst;
    }
    if (n_bad) {
        set_error("pg_batch_solve: " + std::to_string(n_bad) + " RVE(s) did not reach the tolerance");
        return worst;
    }
    return PG_OK;
}

int pg_batch_get_solution(pg_batch* B, int32_t rve, double* U_host) {
    if (!B || !U_host || rve < 0 || rve >= B->n_rve) { set_error("pg_batch_get_solution: invalid argument"); return PG_ERR_ARG; }
    Ctx& c = B->ctx.c;
    cudaSetDevice(c.device);
    const size_t n = 2 * (size_t)(B->noff[rve + 1] - B->noff[rve]);
    PG_CUDA(cudaMemcpyAsync(U_host, c.U + 2 * (size_t)B->noff[rve], n * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    PG_CUDA(cudaStreamSynchronize(c.stream));
    return PG_OK;
}

}  // extern "C"
