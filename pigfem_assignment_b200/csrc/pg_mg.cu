// Geometric multigrid preconditioner for the IGFEM system, and the CG around it (sm_100a).
//
// The reference factors K_ff directly (MUMPS through PETSc,
// src/Solver.cpp:56-142); on the GPU the masked system is solved by CG whose
// preconditioner is one V-cycle over the structured background grid:
//   level 0     the IGFEM system itself (2x2-block CSR, regular + enrichment nodes)
//   level l>0   grid of ceil(n_{l-1}/2) cells per side, 9-point block stencil
// A context made of several RVEs (a batch) has one such hierarchy per RVE, of
// its own depth; every kernel covers all of them, each RVE with its own CG
// scalars, tolerance and end.
//
// Prolongation interpolates the coarse correction bilinearly (in grid index
// space) onto the regular nodes of the finer grid and leaves enrichment
// DOFs to the smoother (their shape functions vanish at the regular nodes,
// so a smooth error lives in the regular DOFs).  Coarse operators are the
// Galerkin products P^T A P of the masked finer operator; a coarse DOF is
// fixed when the finer node at its position is fixed.
//
// Level 0 is smoothed once each way, in two factors: a damped block-Jacobi
// sweep of the regular nodes, and a Chebyshev polynomial of the enrichment
// block (k_mg_enr); before the coarse correction in this order, after it in
// the reverse one, so that the cycle is symmetric.  Both factors reduce the
// error in the energy norm (kOmegaReg and the polynomial's bound), so the
// cycle is positive definite.  Coarse levels take two sweeps of damped block
// Jacobi each way, the coarsest grid (at most 4 cells per side) its inverse.
// Against two sweeps over all of level 0 each way: 74 -> 57 CG iterations at
// 512^2 (rtol 1e-12), each with three products by K instead of five.
//
// A CG iteration is 7 launches and two per coarse level that has more than
// kBottomNodes nodes; it was 43 at 512^2.  Below 512^2 all of them are bound
// by launch and dependent-load latency, above by the reads of K.
//
// Precision: the outer CG always runs in FP64 (operator, vectors, dots and
// the returned residual).  PG_PRECISION_MIXED runs the V-cycle in FP32 (FP32
// copies of every level's operator and FP32 vectors; rows of level 0 are
// summed in FP64); only the preconditioner changes, so the FP64 result and
// its residual are unchanged in kind.
//
// Every kernel of a CG iteration returns at once for an RVE whose "done" flag
// is set, so captured graphs of several iterations may run past convergence
// without changing the result.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "pg_mg_kernels.cuh"

namespace pgb {

using namespace mg;

namespace {

constexpr int kMaxLevels = 16;
constexpr int kChunk = 2;                // CG iterations per graph (the parity of p and r.z is baked in)

// Level vectors in the V-cycle's precision
template <typename T>
struct LevelArrays {
    T *A = nullptr, *Dinv = nullptr;     // 36 and 4 per node: stencil block (dj+1)*3+(di+1), 2x2 row-major
    T *b = nullptr, *x = nullptr, *xo = nullptr;  // 2 per node
};

struct Tiles {
    int4* tile = nullptr;                // RVE, first node column and row, 1 for the RVE's first tile
    int n = 0;
};

struct Level {
    int n = 0;                           // nodes of all RVEs
    int* node_rve = nullptr;             // (several RVEs)
    Pair* pair = nullptr;                // per RVE: the transfer from the finer level
    uint8_t* fixed = nullptr;            // 2 per node
    Tiles down, up;                      // of the transfer to this level, and of this level's post-smoothing
    LevelArrays<double> d;
    LevelArrays<float> f;
};

}  // namespace

struct MgHierarchy {
    int R = 0;                           // RVEs
    int nlev = 0;                        // coarse levels 1..nlev
    std::vector<int> depth;              // and those of each RVE
    Level L[kMaxLevels + 1];
    Spans spans{};
    int n_cta = 0;
    int* node_end = nullptr;             // per RVE
    // enrichment nodes
    int n_enr = 0, n_pieces = 0, max_piece = 0;
    int *enr_node = nullptr, *enr_rve = nullptr;
    Enr enr{};
    unsigned long long* bound = nullptr; // per RVE
    double* coef = nullptr;
    // the bottom of every RVE's cycle
    Bottom* bottom = nullptr;
    Coarse* coarse = nullptr;
    double* XT = nullptr;
    // level-0 vectors of the cycle: x, and the enrichment nodes' after post-smoothing
    double *x0 = nullptr, *x0e = nullptr;
    float *x0f = nullptr, *x0ef = nullptr, *Dinv0f = nullptr;
    bool f32_ready = false;
    // CG: partials (p.q, r.r, r.z), scalars, flags, and their pinned host copies (two slots of flags)
    double *part_pq = nullptr, *part_rr = nullptr, *part_rz = nullptr;
    double* sc = nullptr;
    int* fl = nullptr;
    double* h_sc = nullptr;
    int* h_fl = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaGraphExec_t graph[4] = {};       // of kChunk iterations: FP64 / FP32 cycle, without / with inclusion modes
    // inclusion rigid modes (cohesive meshes): 3 per inclusion, supports disjoint
    int n_inc = 0;                       // 0: no mode space
    int* z_inc = nullptr;                // per node: the inclusion whose modes touch it, -1 none
    double* zval = nullptr;              // per node: [d][k], 2 x 3
    double* E = nullptr;                 // per inclusion: Z_i^T K Z_i (3 x 3)
    double* Einv = nullptr;
    double* w = nullptr;                 // per inclusion: Z_i^T r (3)
    std::vector<void*> owned;
};

namespace {

inline int nb(long long n, int t = kThreads) { return (int)((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// Inclusion rigid modes.  With cohesive interfaces an inclusion whose
// interface has softened can translate and rotate against the matrix at
// little energy; the grid hierarchy cannot represent those discontinuous
// modes (its corrections are continuous), so the preconditioner adds the
// coarse correction Z (Z^T K Z)^-1 Z^T r over them (additively, so it stays
// symmetric positive definite).  Mode k of inclusion i is the rigid motion
// R_k (x translation, y translation, rotation about the centre) inside the
// inclusion and zero outside: R_k at the nodes inside, and at an enrichment
// node the value that makes the field there R_k (inclusion side) or 0
// (matrix side), i.e. minus the parent edge's interpolation of the nodal
// values.  Distinct inclusions share no element, so Z^T K Z is block
// diagonal with one 3 x 3 block per inclusion.
// ---------------------------------------------------------------------------
__global__ void k_modes_E(int n, const int* __restrict__ z_inc, const double* __restrict__ zval,
                          const int* __restrict__ row_ptr, const int* __restrict__ col, const double* __restrict__ K,
                          const uint8_t* __restrict__ fixed, double* E) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int zi = z_inc[q];
    if (zi < 0) return;
    double y[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    for (int p = row_ptr[q]; p < row_ptr[q + 1]; ++p) {
        const int cn = col[p];
        if (z_inc[cn] != zi) continue;
        const double* blk = K + 4 * (size_t)p;
        for (int d = 0; d < 2; ++d)
            for (int e = 0; e < 2; ++e) {
                if (fixed[2 * cn + e]) continue;
                const double kde = blk[2 * d + e];
                for (int l = 0; l < 3; ++l) y[d][l] += kde * zval[6 * (size_t)cn + 3 * e + l];
            }
    }
    for (int k = 0; k < 3; ++k)
        for (int l = 0; l < 3; ++l) {
            double v = 0.0;
            for (int d = 0; d < 2; ++d)
                if (!fixed[2 * q + d]) v += zval[6 * (size_t)q + 3 * d + k] * y[d][l];
            atomicAdd(&E[9 * zi + 3 * k + l], v);
        }
}

// 3 x 3 inverse per inclusion (zero when the block is numerically singular)
__global__ void k_modes_inv(int n_inc, const double* E, double* Einv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_inc) return;
    const double* a = E + 9 * i;
    const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8], c02 = a[3] * a[7] - a[4] * a[6];
    const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
    double scale = 0.0;
    for (int k = 0; k < 9; ++k) scale = fmax(scale, fabs(a[k]));
    double* o = Einv + 9 * i;
    if (!(fabs(det) > 1e-13 * scale * scale * scale)) {
        for (int k = 0; k < 9; ++k) o[k] = 0.0;
        return;
    }
    const double r = 1.0 / det;
    o[0] = c00 * r;
    o[1] = (a[2] * a[7] - a[1] * a[8]) * r;
    o[2] = (a[1] * a[5] - a[2] * a[4]) * r;
    o[3] = c01 * r;
    o[4] = (a[0] * a[8] - a[2] * a[6]) * r;
    o[5] = (a[2] * a[3] - a[0] * a[5]) * r;
    o[6] = c02 * r;
    o[7] = (a[1] * a[6] - a[0] * a[7]) * r;
    o[8] = (a[0] * a[4] - a[1] * a[3]) * r;
}

__global__ void k_modes_zero(int n, double* w, const int* done) {
    if (done && done[0]) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) w[i] = 0.0;
}

// w_i = Z_i^T r
__global__ void k_modes_dot(int n, const int* __restrict__ z_inc, const double* __restrict__ zval,
                            const uint8_t* __restrict__ fixed, const double* __restrict__ r, double* w, const int* done) {
    if (done && done[0]) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int zi = z_inc[q];
    if (zi < 0) return;
    const double r0 = fixed[2 * q] ? 0.0 : r[2 * q], r1 = fixed[2 * q + 1] ? 0.0 : r[2 * q + 1];
    for (int k = 0; k < 3; ++k)
        atomicAdd(&w[3 * zi + k], zval[6 * (size_t)q + k] * r0 + zval[6 * (size_t)q + 3 + k] * r1);
}

// z += Z_i E_i^-1 w_i
__global__ void k_modes_add(int n, const int* __restrict__ z_inc, const double* __restrict__ zval,
                            const uint8_t* __restrict__ fixed, const double* __restrict__ Einv,
                            const double* __restrict__ w, double* z, const int* done) {
    if (done && done[0]) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int zi = z_inc[q];
    if (zi < 0) return;
    const double* B = Einv + 9 * zi;
    const double* wi = w + 3 * zi;
    double cc[3];
    for (int k = 0; k < 3; ++k) cc[k] = B[3 * k] * wi[0] + B[3 * k + 1] * wi[1] + B[3 * k + 2] * wi[2];
    for (int d = 0; d < 2; ++d) {
        if (fixed[2 * q + d]) continue;
        z[2 * q + d] += zval[6 * (size_t)q + 3 * d] * cc[0] + zval[6 * (size_t)q + 3 * d + 1] * cc[1] +
                        zval[6 * (size_t)q + 3 * d + 2] * cc[2];
    }
}


// ---------------------------------------------------------------------------
// Structure (once per mesh)
// ---------------------------------------------------------------------------
template <typename T>
int mg_alloc(MgHierarchy& m, T** p, size_t n) {
    *p = nullptr;
    PG_CUDA(cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(T)));
    m.owned.push_back((void*)*p);
    return PG_OK;
}

template <typename T>
int mg_upload(MgHierarchy& m, T** p, const std::vector<T>& v) {
    const int rc = mg_alloc(m, p, v.size());
    if (rc) return rc;
    if (!v.empty()) PG_CUDA(h2d_sync(*p, v.data(), v.size() * sizeof(T)));
    return PG_OK;
}

// Device memory of many arrays in one allocation (each 256-byte aligned): a
// hierarchy has some sixty, and an allocation each took longer than a solve.
struct Arena {
    struct Item {
        void** p;
        size_t bytes;
        const void* src;
    };
    std::vector<Item> items;
    template <typename T>
    void add(T** p, size_t n) {
        items.push_back({(void**)p, std::max<size_t>(n, 1) * sizeof(T), nullptr});
    }
    // with contents (kept by the caller until commit)
    template <typename T>
    void add(T** p, const std::vector<T>& v) {
        items.push_back({(void**)p, std::max<size_t>(v.size(), 1) * sizeof(T), v.empty() ? nullptr : v.data()});
    }
    int commit(MgHierarchy& m) {
        size_t total = 0;
        for (const Item& it : items) total += (it.bytes + 255) & ~size_t(255);
        char* base = nullptr;
        int rc = mg_alloc(m, &base, total);
        if (rc) return rc;
        for (const Item& it : items) {
            *it.p = base;
            if (it.src) PG_CUDA(cudaMemcpy(base, it.src, it.bytes, cudaMemcpyHostToDevice));
            base += (it.bytes + 255) & ~size_t(255);
        }
        PG_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
        items.clear();
        return PG_OK;
    }
};

// Inclusion rigid modes of a cohesive mesh (host, once per mesh).
int modes_build(Ctx& c, MgHierarchy& m) {
    const HostMesh& hm = c.hm;
    const int ni = (int)hm.spec.inclusions.size();
    if (!hm.spec.cohesive || ni == 0) return PG_OK;
    const int nn = hm.n_nodes();
    // side of every enrichment node: 1 if an inclusion-material child uses it, 0 if a matrix child does
    std::vector<int> side(hm.n_enr, -1);
    for (int ci = 0; ci < hm.n_cut; ++ci) {
        const CutTemplate& T = cut_template(hm.cut_tmpl[ci]);
        for (int ch = 0; ch < T.n_child; ++ch) {
            const int mat = hm.cut_child_mat[(size_t)ci * kMaxChildren + ch];
            for (int k = 0; k < T.child_n[ch]; ++k) {
                const int ln = T.child_nodes[ch][k];
                if (ln < 3) continue;
                const int node = hm.cut_enr[(size_t)ci * kMaxEnr + ln - 3];
                if (node >= hm.n_reg) side[node - hm.n_reg] = mat == hm.spec.matrix_mat ? 0 : 1;
            }
        }
    }
    std::vector<int> zinc(nn, -1);
    std::vector<double> zval(6 * (size_t)nn, 0.0);
    auto rigid = [&](int i, double x, double y, double out[2][3]) {
        const Inclusion& I = hm.spec.inclusions[i];
        out[0][0] = 1.0; out[0][1] = 0.0; out[0][2] = -(y - I.cy);
        out[1][0] = 0.0; out[1][1] = 1.0; out[1][2] = x - I.cx;
    };
    for (int n = 0; n < hm.n_reg; ++n) {
        const int i = hm.node_detect[n];
        if (i < 0 || i >= ni) continue;
        double R[2][3];
        rigid(i, hm.x[n], hm.y[n], R);
        zinc[n] = i;
        for (int d = 0; d < 2; ++d)
            for (int k = 0; k < 3; ++k) zval[6 * (size_t)n + 3 * d + k] = R[d][k];
    }
    for (int k = 0; k < hm.n_enr; ++k) {
        const int n = hm.n_reg + k, i = hm.enr_inc[k];
        if (i < 0 || i >= ni || side[k] < 0) continue;
        const int a = hm.enr_edge[2 * k], b = hm.enr_edge[2 * k + 1];
        const double ex = hm.x[b] - hm.x[a], ey = hm.y[b] - hm.y[a];
        const double t = ((hm.x[n] - hm.x[a]) * ex + (hm.y[n] - hm.y[a]) * ey) / (ex * ex + ey * ey);
        double Ra[2][3] = {}, Rb[2][3] = {}, Rn[2][3] = {};
        if (hm.node_detect[a] == i) rigid(i, hm.x[a], hm.y[a], Ra);
        if (hm.node_detect[b] == i) rigid(i, hm.x[b], hm.y[b], Rb);
        if (side[k] == 1) rigid(i, hm.x[n], hm.y[n], Rn);
        zinc[n] = i;
        for (int d = 0; d < 2; ++d)
            for (int q = 0; q < 3; ++q)
                zval[6 * (size_t)n + 3 * d + q] = Rn[d][q] - ((1.0 - t) * Ra[d][q] + t * Rb[d][q]);
    }
    int rc;
    if ((rc = mg_upload(m, &m.z_inc, zinc)) || (rc = mg_upload(m, &m.zval, zval)) || (rc = mg_alloc(m, &m.E, 9 * (size_t)ni)) ||
        (rc = mg_alloc(m, &m.Einv, 9 * (size_t)ni)) || (rc = mg_alloc(m, &m.w, 3 * (size_t)ni)))
        return rc;
    m.n_inc = ni;
    return PG_OK;
}

// The enrichment pieces of one RVE (see k_mg_enr): its enrichment nodes in
// depth-first order of the K_ee graph (along the interfaces), cut into cores
// of kPieceRows; around each core the nodes within kChebSteps - 1 steps.
struct RvePieces {
    std::vector<Piece> piece;
    std::vector<int> node, eptr;
    std::vector<int2> ent;
};

void build_pieces(const HostMesh& hm, int rve, int lo, int hi, RvePieces& out) {
    const int n = hi - lo;
    std::vector<int> order, stack, local(n, -1), rep(n);
    std::vector<char> seen(n, 0);
    order.reserve(n);
    // a node and its mirror across a cohesive interface (the same place) follow each other in the order, so that
    // a core spans the interface instead of one side of it (108 against 60 local rows)
    for (int v = 0; v < n; ++v) {
        rep[v] = v;
        for (int q = hm.row_ptr[lo + v]; q < hm.row_ptr[lo + v + 1]; ++q) {
            const int j = hm.col[q];
            if (j >= lo && j < lo + v && hm.x[j] == hm.x[lo + v] && hm.y[j] == hm.y[lo + v]) {
                rep[v] = rep[j - lo];
                break;
            }
        }
    }
    auto visit = [&](int v) {
        seen[v] = 1;
        order.push_back(v);
        for (int q = hm.row_ptr[lo + v + 1] - 1; q >= hm.row_ptr[lo + v]; --q) {
            const int j = hm.col[q] - lo;
            if (j >= 0 && j < n && !seen[j] && rep[j] != rep[v]) stack.push_back(j);
        }
    };
    for (int s = 0; s < n; ++s) {
        if (seen[s]) continue;
        stack.push_back(s);
        while (!stack.empty()) {
            const int v = stack.back();
            stack.pop_back();
            if (seen[v]) continue;
            visit(v);
            for (int q = hm.row_ptr[lo + v]; q < hm.row_ptr[lo + v + 1]; ++q) {
                const int j = hm.col[q] - lo;
                if (j >= 0 && j < n && !seen[j] && rep[j] == rep[v]) visit(j);
            }
        }
    }
    std::vector<int> loc;
    for (int c0 = 0; c0 < n; c0 += kPieceRows) {
        Piece p{};
        p.rve = rve;
        p.row0 = (int)out.node.size();
        loc.assign(order.begin() + c0, order.begin() + std::min(n, c0 + kPieceRows));
        for (size_t k = 0; k < loc.size(); ++k) local[loc[k]] = (int)k;
        p.end[0] = (int)loc.size();
        for (int d = 1; d < kChebSteps; ++d) {
            const int b = d == 1 ? 0 : p.end[d - 2], e = p.end[d - 1];
            for (int k = b; k < e; ++k)
                for (int q = hm.row_ptr[lo + loc[k]]; q < hm.row_ptr[lo + loc[k] + 1]; ++q) {
                    const int j = hm.col[q];
                    if (j < lo || j >= hi || local[j - lo] >= 0) continue;
                    local[j - lo] = (int)loc.size();
                    loc.push_back(j - lo);
                }
            p.end[d] = (int)loc.size();
        }
        for (size_t k = 0; k < loc.size(); ++k) {
            out.node.push_back(lo + loc[k]);
            out.eptr.push_back((int)out.ent.size());
            if ((int)k >= p.end[kChebSteps - 2]) continue;  // the outermost ring only starts the recurrence
            for (int q = hm.row_ptr[lo + loc[k]]; q < hm.row_ptr[lo + loc[k] + 1]; ++q) {
                const int j = hm.col[q];
                if (j >= lo && j < hi) out.ent.push_back(make_int2(q, local[j - lo]));
            }
        }
        for (int v : loc) local[v] = -1;
        out.piece.push_back(p);
    }
}

int build_hierarchy(Ctx& c) {
    const HostMesh& hm = c.hm;
    const int R = (int)hm.grids.size();
    if (R < 1) {
        set_error("multigrid: mesh without a structured background grid");
        return PG_ERR_ARG;
    }
    if (!c.grid_emat) {  // (no builder makes one: their rows begin with the grid neighbours, see grid_pattern_ok)
        set_error("multigrid: the background grid's rows are not laid out as its Galerkin product reads them");
        return PG_ERR_ARG;
    }
    // each RVE's grids, coarsened until both sides have at most kCoarseCells cells
    std::vector<std::vector<std::pair<int, int>>> dims(R);
    int nlev = 0;
    for (int r = 0; r < R; ++r) {
        int nx = hm.grids[r].nx, ny = hm.grids[r].ny;
        dims[r].push_back({nx, ny});
        while ((nx > kCoarseCells || ny > kCoarseCells) && (int)dims[r].size() <= kMaxLevels) {
            nx = (nx + 1) / 2;
            ny = (ny + 1) / 2;
            dims[r].push_back({nx, ny});
        }
        if (dims[r].size() < 2 || nx > kCoarseCells || ny > kCoarseCells) {
            set_error("multigrid: grid too small or too large to coarsen");
            return PG_ERR_ARG;
        }
        nlev = std::max(nlev, (int)dims[r].size() - 1);
    }
    auto nodes = [&](int r, int l) { return (dims[r][l].first + 1) * (dims[r][l].second + 1); };
    MgHierarchy* mp = new MgHierarchy();
    c.mg = mp;
    MgHierarchy& m = *mp;
    m.R = R;
    m.nlev = nlev;
    for (const auto& d : dims) m.depth.push_back((int)d.size() - 1);
    Arena ar;
    // the bottom of each RVE's cycle: its levels of at most kBottomNodes nodes, as many as its threads own
    std::vector<Bottom> bottom(R);
    std::vector<int> kb(R);
    for (int r = 0; r < R; ++r) {
        const int depth = (int)dims[r].size() - 1;
        int k = depth, threads = 0, vec = nodes(r, depth);
        while (k > 1 && depth - k + 1 < kBottomLevels && nodes(r, k - 1) <= kBottomNodes) {
            threads += (nodes(r, k - 1) + 31) / 32 * 32;
            vec += nodes(r, k - 1);
            if (threads > kBottomThreads || vec > kBottomVec) break;
            --k;
        }
        kb[r] = k;
    }
    // levels: offsets, transfers, tiles
    std::vector<std::vector<int>> off(nlev + 1, std::vector<int>(R, 0));
    std::vector<std::vector<Pair>> pairs(nlev + 1);
    std::vector<std::vector<int4>> down(nlev + 1), up(nlev + 1);
    std::vector<std::vector<int>> node_rve(nlev + 1);
    for (int r = 0; r < R; ++r) off[0][r] = hm.grids[r].node_off;
    for (int l = 1; l <= nlev; ++l) {
        Level& L = m.L[l];
        pairs[l].assign(R, Pair{0, 0, 0, 0, -1, -1});
        for (int r = 0; r < R; ++r) {
            if ((int)dims[r].size() <= l) continue;
            off[l][r] = L.n;
            const int nx = dims[r][l].first, ny = dims[r][l].second;
            pairs[l][r] = Pair{off[l - 1][r], dims[r][l - 1].first, dims[r][l - 1].second, L.n, nx, ny};
            if (R > 1) node_rve[l].insert(node_rve[l].end(), nodes(r, l), r);
            L.n += nodes(r, l);
            if (l <= kb[r])
                for (int J = 0; J <= ny; J += kDownTile)
                    for (int I = 0; I <= nx; I += kDownTile) down[l].push_back(make_int4(r, I, J, I == 0 && J == 0));
            if (l < kb[r])
                for (int J = 0; J <= ny; J += kUpTile)
                    for (int I = 0; I <= nx; I += kUpTile) up[l].push_back(make_int4(r, I, J, 0));
        }
        L.down.n = (int)down[l].size();
        L.up.n = (int)up[l].size();
        ar.add(&L.pair, pairs[l]);
        ar.add(&L.down.tile, down[l]);
        ar.add(&L.up.tile, up[l]);
        if (R > 1) ar.add(&L.node_rve, node_rve[l]);
        ar.add(&L.fixed, 2 * (size_t)L.n);
        ar.add(&L.d.A, 36 * (size_t)L.n);
        ar.add(&L.d.Dinv, 4 * (size_t)L.n);
        for (double** v : {&L.d.b, &L.d.x, &L.d.xo}) ar.add(v, 2 * (size_t)L.n);
    }
    for (int r = 0; r < R; ++r) {
        const int depth = (int)dims[r].size() - 1;
        Bottom& B = bottom[r];
        B = Bottom{};
        B.first = kb[r];
        B.nlev = depth - kb[r] + 1;
        for (int k = 0; k < B.nlev; ++k) {
            B.nx[k] = dims[r][kb[r] + k].first;
            B.ny[k] = dims[r][kb[r] + k].second;
            B.off[k] = off[kb[r] + k][r];
            const int n = nodes(r, kb[r] + k);
            if (k + 1 < B.nlev) B.thread[k + 1] = B.thread[k] + (n + 31) / 32 * 32;
            if (k + 1 < B.nlev) B.vec[k + 1] = B.vec[k] + n;
        }
        B.foff = off[kb[r] - 1][r];
        B.fnx = dims[r][kb[r] - 1].first;
        B.fny = dims[r][kb[r] - 1].second;
    }
    // row spans of the level-0 kernels: as many CTAs as the GPU holds, each with about as many blocks of K, in
    // steps of kStep rows
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    constexpr int kStep = 16;
    const long long total = hm.n_blocks() + 2LL * c.n_nodes;
    const double per_cta = std::max((double)total / (sms * kSpanCtasPerSm), 1.0);
    std::vector<int4> span;
    std::vector<int2> range(R);
    std::vector<int> reg_end(R), node_end(R);
    for (int r = 0; r < R; ++r) {
        const auto& gb = hm.grids[r];
        const int lo = gb.node_off, hi = r + 1 < R ? hm.grids[r + 1].node_off : c.n_nodes;
        reg_end[r] = lo + gb.n_reg;
        node_end[r] = hi;
        range[r].x = (int)span.size();
        int row = lo;
        while (row < hi) {
            int end = row;
            double w = 0.0;
            while (end < hi && (end == row || w + 0.5 * (hm.row_ptr[std::min(end + kStep, hi)] - hm.row_ptr[end]) < per_cta)) {
                const int e = std::min(end + kStep, hi);
                w += hm.row_ptr[e] - hm.row_ptr[end] + 2.0 * (e - end);
                end = e;
            }
            span.push_back(make_int4(r, row, end, 0));
            row = end;
        }
        range[r].y = (int)span.size();
    }
    m.n_cta = (int)span.size();
    int4* d_span;
    int2* d_range;
    int* d_reg;
    ar.add(&d_span, span);
    ar.add(&d_range, range);
    ar.add(&d_reg, reg_end);
    ar.add(&m.node_end, node_end);
    // enrichment pieces, RVE by RVE in parallel
    std::vector<RvePieces> rp(R);
    parallel_for(R, 1, [&](long long r) { build_pieces(hm, (int)r, reg_end[r], node_end[r], rp[r]); });
    std::vector<Piece> piece;
    std::vector<int> pnode, peptr, enr_node, enr_rve;
    std::vector<int2> pent;
    for (int r = 0; r < R; ++r) {
        const int n0 = (int)pnode.size(), e0 = (int)pent.size();
        for (Piece p : rp[r].piece) {
            p.row0 += n0;
            m.max_piece = std::max(m.max_piece, p.end[kChebSteps - 1]);
            piece.push_back(p);
        }
        pnode.insert(pnode.end(), rp[r].node.begin(), rp[r].node.end());
        for (int e : rp[r].eptr) peptr.push_back(e + e0);
        pent.insert(pent.end(), rp[r].ent.begin(), rp[r].ent.end());
        for (int i = reg_end[r]; i < node_end[r]; ++i) {
            enr_node.push_back(i);
            enr_rve.push_back(r);
        }
    }
    peptr.push_back((int)pent.size());
    m.n_pieces = (int)piece.size();
    m.n_enr = (int)enr_node.size();
    Piece* d_piece;
    int *d_pnode, *d_peptr;
    int2* d_pent;
    ar.add(&d_piece, piece);
    ar.add(&d_pnode, pnode);
    ar.add(&d_peptr, peptr);
    ar.add(&d_pent, pent);
    ar.add(&m.enr_node, enr_node);
    ar.add(&m.enr_rve, enr_rve);
    ar.add(&m.bound, (size_t)R);
    ar.add(&m.coef, (size_t)kChebCoef * R);
    ar.add(&m.bottom, bottom);
    std::vector<Coarse> coarse(R);  // (device pointers are known after the commit)
    ar.add(&m.coarse, (size_t)R);
    ar.add(&m.XT, (size_t)kCoarseStride * R);
    ar.add(&m.x0, (size_t)c.n_dof);
    ar.add(&m.x0e, (size_t)c.n_dof);
    for (double** v : {&m.part_pq, &m.part_rr, &m.part_rz}) ar.add(v, (size_t)m.n_cta);
    ar.add(&m.sc, (size_t)kScal * R);
    ar.add(&m.fl, (size_t)kFlags * R);
    int rc = ar.commit(m);
    if (rc) return rc;
    m.spans = Spans{d_span, d_range, d_reg};
    m.enr = Enr{d_piece, d_pnode, d_peptr, d_pent, m.coef};
    for (int r = 0; r < R; ++r) {
        const int l = (int)dims[r].size() - 1;
        coarse[r] = Coarse{m.L[l].d.A, m.L[l].fixed, off[l][r], dims[r][l].first, dims[r][l].second, 0};
    }
    PG_CUDA(h2d_sync(m.coarse, coarse.data(), coarse.size() * sizeof(Coarse)));
    PG_CUDA(cudaMallocHost((void**)&m.h_sc, (size_t)kScal * R * sizeof(double)));
    PG_CUDA(cudaMallocHost((void**)&m.h_fl, 2 * (size_t)kFlags * R * sizeof(int)));
    for (cudaEvent_t& e : m.ev) PG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    // kernels whose shared memory exceeds the default (the attribute belongs to the device, so the largest any
    // hierarchy on it may ask for)
    if ((size_t)m.max_piece * 8 * sizeof(double) > 100 * 1024) {
        set_error("multigrid: enrichment piece too large for shared memory");
        return PG_ERR_LIMIT;
    }
    PG_CUDA(cudaFuncSetAttribute(k_mg_bottom<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 4 * kBottomStride * (int)sizeof(Vec2<double>)));
    PG_CUDA(cudaFuncSetAttribute(k_mg_bottom<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 4 * kBottomStride * (int)sizeof(Vec2<float>)));
    for (auto k : {k_mg_enr<double, false, kPieceThreads>, k_mg_enr<double, true, kPieceThreads>})
        PG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    for (auto k : {k_mg_enr<float, false, kPieceThreads>, k_mg_enr<float, true, kPieceThreads>,
                   k_mg_enr<float, false, kPieceThreadsWide>, k_mg_enr<float, true, kPieceThreadsWide>})
        PG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    // coarse masks by injection
    cudaStream_t s = c.stream;
    const uint8_t* ff = c.fixed;
    for (int l = 1; l <= nlev; ++l) {
        Level& L = m.L[l];
        k_mg_inject_mask<<<nb(L.n), kThreads, 0, s>>>(L.n, L.node_rve, L.pair, ff, L.fixed);
        ff = L.fixed;
    }
    PG_CUDA(cudaGetLastError());
    PG_CUDA(cudaStreamSynchronize(s));
    return R == 1 ? modes_build(c, m) : PG_OK;
}

// the FP32 cycle's arrays, on its first use
int ensure_f32(Ctx& c, MgHierarchy& m) {
    if (m.f32_ready) return PG_OK;
    Arena ar;
    for (int l = 1; l <= m.nlev; ++l) {
        Level& L = m.L[l];
        ar.add(&L.f.A, 36 * (size_t)L.n);
        ar.add(&L.f.Dinv, 4 * (size_t)L.n);
        for (float** v : {&L.f.b, &L.f.x, &L.f.xo}) ar.add(v, 2 * (size_t)L.n);
    }
    ar.add(&m.x0f, (size_t)c.n_dof);
    ar.add(&m.x0ef, (size_t)c.n_dof);
    ar.add(&m.Dinv0f, 4 * (size_t)c.n_nodes);
    const int rc = ar.commit(m);
    if (rc == PG_OK) m.f32_ready = true;
    return rc;
}

// Numeric set-up for the current K (every solve: K changes between Newton iterations).
int mg_numeric(Ctx& c, bool f32, bool modes, cudaStream_t s) {
    MgHierarchy& m = *c.mg;
    const int n0 = c.n_nodes;
    int rc;
    if (f32 && (rc = ensure_f32(c, m))) return rc;
    cudaMemsetAsync(m.fl, 0, (size_t)kFlags * m.R * sizeof(int), s);
    // level 0: block Jacobi of the masked K, and the enrichment block's polynomial
    k_prec_setup<double><<<nb(n0), kThreads, 0, s>>>(n0, c.diag, c.K, c.fixed, 1, 0, c.minv);
    if (f32) {
        launch_to_fp32(c, s);
        k_mg_to_f32<<<nb(4LL * n0), kThreads, 0, s>>>(4 * (size_t)n0, c.minv, m.Dinv0f);
    }
    if (m.n_enr > 0) {
        cudaMemsetAsync(m.bound, 0, (size_t)m.R * sizeof(unsigned long long), s);
        k_enr_bound<<<nb(m.n_enr, 128), 128, 0, s>>>(m.n_enr, m.enr_node, m.enr_rve, m.spans.reg_end, m.node_end, c.row_ptr,
                                                      c.col, c.diag, c.K, m.bound);
        k_enr_coef<<<nb(m.R), kThreads, 0, s>>>(m.R, m.bound, m.coef);
    }
    for (int l = 1; l <= m.nlev; ++l) {
        Level& L = m.L[l];
        const uint8_t* ff = l > 1 ? m.L[l - 1].fixed : c.fixed;
        float* Af = f32 ? L.f.A : nullptr;
        float* Df = f32 ? L.f.Dinv : nullptr;
        if (l == 1)
            k_mg_galerkin<true><<<nb(L.n, kGalNodes), kGalThreads, 0, s>>>(L.n, L.node_rve, L.pair, c.row_ptr, c.K,
                                                                           nullptr, ff, L.fixed, L.d.A, Af, L.d.Dinv, Df);
        else
            k_mg_galerkin<false><<<nb(L.n, kGalNodes), kGalThreads, 0, s>>>(L.n, L.node_rve, L.pair, nullptr, nullptr,
                                                                            m.L[l - 1].d.A, ff, L.fixed, L.d.A, Af, L.d.Dinv,
                                                                            Df);
    }
    if (m.n_inc > 0 && modes) {
        cudaMemsetAsync(m.E, 0, 9 * (size_t)m.n_inc * sizeof(double), s);
        k_modes_E<<<nb(n0), kThreads, 0, s>>>(n0, m.z_inc, m.zval, c.row_ptr, c.col, c.K, c.fixed, m.E);
        k_modes_inv<<<nb(m.n_inc), kThreads, 0, s>>>(m.n_inc, m.E, m.Einv);
    }
    k_mg_coarse_inverse<<<m.R, kFactorThreads, 0, s>>>(m.coarse, m.XT, m.fl);
    PG_CUDA(cudaGetLastError());
    return PG_OK;
}

// What the V-cycle's precision decides: the level-0 operator and vectors and the levels' arrays
template <typename T>
struct Cycle;
template <>
struct Cycle<double> {
    static const double* K(const Ctx& c) { return c.K; }
    static const double* Dinv(const Ctx& c, const MgHierarchy&) { return c.minv; }
    static double* x(const MgHierarchy& m) { return m.x0; }
    static double* xe(const MgHierarchy& m) { return m.x0e; }
    static LevelArrays<double>& lev(Level& L) { return L.d; }
};
template <>
struct Cycle<float> {
    static const float* K(const Ctx& c) { return c.Kf; }
    static const float* Dinv(const Ctx&, const MgHierarchy& m) { return m.Dinv0f; }
    static float* x(const MgHierarchy& m) { return m.x0f; }
    static float* xe(const MgHierarchy& m) { return m.x0ef; }
    static LevelArrays<float>& lev(Level& L) { return L.f; }
};

// The enrichment nodes' smoothing: x_e of the cycle's x into xout.  Pieces of
// a cohesive mesh hold some 100 rows (both sides of an interface) and get a
// thread group per row in the FP32 cycle; in FP64 a row's blocks leave no
// registers for that.
template <typename T, bool POST>
void mg_enr(Ctx& c, MgHierarchy& m, cudaStream_t s, const double* r, T* xout, const int* fl) {
    using C = Cycle<T>;
    if (m.n_pieces == 0) return;
    auto go = [&](auto kern, int threads) {
        launch_pdl(kern, m.n_pieces, threads, (size_t)m.max_piece * 4 * sizeof(Vec2<T>), s, m.enr, c.row_ptr, c.col, C::K(c),
                   C::Dinv(c, m), c.fixed, m.spans.reg_end, r, C::x(m), xout, fl);
    };
    if constexpr (std::is_same<T, float>::value) {
        if (m.max_piece > kPieceThreads / kRowLanes) {
            go(k_mg_enr<T, POST, kPieceThreadsWide>, kPieceThreadsWide);
            return;
        }
    }
    go(k_mg_enr<T, POST, kPieceThreads>, kPieceThreads);
}

// The V-cycle after its first sweep (which CG's update has formed): z = V(r)
// and the partials of r.z.  fl null outside CG; check: this cycle follows a
// CG update, whose r.r it tests.
template <typename T>
void mg_cycle(Ctx& c, MgHierarchy& m, bool modes, cudaStream_t s, const double* r, double* z, int* fl, bool check) {
    using C = Cycle<T>;
    const T *K = C::K(c), *D0 = C::Dinv(c, m);
    T *x0 = C::x(m), *xe = C::xe(m);
    mg_enr<T, false>(c, m, s, r, x0, fl);
    launch_pdl(k_mg_down0<T>, m.L[1].down.n, kDown0Threads, 0, s, m.L[1].down.tile, m.L[1].pair, c.row_ptr, c.col, K, c.fixed, r, x0,
                                                         m.L[1].fixed, C::lev(m.L[1]).b, m.spans, m.part_rr, m.sc, fl,
                                                         check ? 1 : 0);
    for (int l = 2; l <= m.nlev && m.L[l].down.n > 0; ++l) {
        Level &F = m.L[l - 1], &L = m.L[l];
        LevelArrays<T>& f = C::lev(F);
        launch_pdl(k_mg_down<T>, L.down.n, kTileThreads, 0, s, L.down.tile, L.pair, f.A, f.Dinv, f.b, f.x, L.fixed,
                                                       C::lev(L).b, fl);
    }
    BottomArrays<T> ba{};
    for (int l = 1; l <= m.nlev; ++l) {
        LevelArrays<T>& v = C::lev(m.L[l]);
        ba.A[l] = v.A;
        ba.Dinv[l] = v.Dinv;
        ba.fixed[l] = m.L[l].fixed;
        ba.b[l] = v.b;
        ba.xo[l] = v.xo;
    }
    launch_pdl(k_mg_bottom<T>, m.R, kBottomThreads, 4 * kBottomStride * sizeof(Vec2<T>), s, m.bottom, ba, m.XT, c.fixed, x0, fl);
    for (int l = m.nlev - 1; l >= 1; --l) {
        Level& L = m.L[l];
        if (L.up.n == 0) continue;
        LevelArrays<T>& v = C::lev(L);
        const T* xc = C::lev(m.L[l + 1]).xo;
        if (l == 1)
            launch_pdl(k_mg_up<T, true>, L.up.n, kTileThreads, 0, s, L.up.tile, L.pair, m.L[2].pair, v.A, v.Dinv, L.fixed, v.b, v.x, xc,
                                                             nullptr, c.fixed, x0, fl);
        else
            launch_pdl(k_mg_up<T, false>, L.up.n, kTileThreads, 0, s, L.up.tile, L.pair, m.L[l + 1].pair, v.A, v.Dinv, L.fixed, v.b,
                                                              v.x, xc, v.xo, nullptr, nullptr, fl);
    }
    mg_enr<T, true>(c, m, s, r, xe, fl);
    launch_pdl(k_mg_post<T>, m.n_cta, kSpanThreads, 0, s, m.spans, c.row_ptr, c.col, K, D0, c.fixed, r, x0, xe, z, fl, m.part_rz);
    if (m.n_inc > 0 && modes) {
        const int n = c.n_nodes;
        k_modes_zero<<<nb(3 * m.n_inc), kThreads, 0, s>>>(3 * m.n_inc, m.w, fl);
        k_modes_dot<<<nb(n), kThreads, 0, s>>>(n, m.z_inc, m.zval, c.fixed, r, m.w, fl);
        k_modes_add<<<nb(n), kThreads, 0, s>>>(n, m.z_inc, m.zval, c.fixed, m.Einv, m.w, z, fl);
        launch_pdl(k_cg_dot, m.n_cta, kSpanThreads, 0, s, m.spans, r, z, fl, m.part_rz);
    }
}

// kChunk CG iterations
template <typename T>
void cg_iterations(Ctx& c, MgHierarchy& m, bool modes, cudaStream_t s) {
    double* pb[2] = {c.p, c.xi};
    for (int it = 0; it < kChunk; ++it) {
        const int P = it & 1;
        launch_pdl(k_cg_spmv, m.n_cta, kSpanThreads, 0, s, m.spans, c.row_ptr, c.col, c.K, c.fixed, c.z, pb[1 - P], pb[P], c.q,
                                                   m.part_rz, m.sc, m.fl, m.part_pq, P);
        launch_pdl(k_cg_update<T>, m.n_cta, kSpanThreads, 0, s, m.spans, c.dx, c.r, pb[P], c.q, Cycle<T>::Dinv(c, m), Cycle<T>::x(m),
                                                        m.part_pq, m.sc, m.fl, m.part_rr, P);
        mg_cycle<T>(c, m, modes, s, c.r, c.z, m.fl, true);
    }
}

// CG on mask(K) dx = mask(b) (b = c.b, dx = c.dx) for every RVE; the host
// copies of the flags and scalars are current when it returns PG_OK.
template <typename T>
int cg_run(Ctx& c, MgHierarchy& m, bool modes, const pg_solver_cfg& cfg, cudaStream_t s) {
    const bool f32 = std::is_same<T, float>::value;
    const size_t fl_bytes = (size_t)kFlags * m.R * sizeof(int);
    int rc = mg_numeric(c, f32, modes, s);
    if (rc) return rc;
    launch_pdl(k_cg_start<T>, m.n_cta, kSpanThreads, 0, s, m.spans, c.fixed, c.b, c.r, c.dx, Cycle<T>::Dinv(c, m), Cycle<T>::x(m),
                                                   m.part_rr);
    launch_pdl(k_cg_tol, m.R, kSpanThreads, 0, s, m.spans, m.part_rr, cfg.rtol * cfg.rtol, m.sc, m.fl);
    cudaMemsetAsync(c.xi, 0, (size_t)c.n_dof * sizeof(double), s);  // p before the first iteration
    mg_cycle<T>(c, m, modes, s, c.r, c.z, nullptr, false);
    PG_CUDA(cudaGetLastError());
    cudaMemcpyAsync(m.h_sc, m.sc, (size_t)kScal * m.R * sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(m.h_fl, m.fl, fl_bytes, cudaMemcpyDeviceToHost, s);
    cudaGraphExec_t& exec = m.graph[(f32 ? 1 : 0) + (modes ? 2 : 0)];
    if (!exec && cfg.max_iter > 0) {
        // every pointer in it belongs to the context, so one graph serves all its solves
        cudaGraph_t graph;
        PG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        cg_iterations<T>(c, m, modes, s);
        // (a graph that lacks a refused launch would be kept for every later solve)
        const cudaError_t le = cudaGetLastError();
        PG_CUDA(cudaStreamEndCapture(s, &graph));
        const cudaError_t ie = le != cudaSuccess ? le : cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) {
            exec = nullptr;
            return cuda_fail(ie, "multigrid CG graph");
        }
    }
    PG_CUDA(cudaStreamSynchronize(s));
    for (int r = 0; r < m.R; ++r)
        if (m.h_fl[kFlags * r + 3]) {
            set_error("multigrid: singular coarsest operator");
            return PG_ERR_BREAKDOWN;
        }
    auto all_done = [&](const int* f) {
        for (int r = 0; r < m.R; ++r)
            if (!f[kFlags * r]) return false;
        return true;
    };
    int* slot[2] = {m.h_fl, m.h_fl + kFlags * m.R};
    int launched = 0, last = 0;
    if (!all_done(slot[0])) {
        // the next graph is in flight while the host looks at the last one's flags
        while (launched < cfg.max_iter) {
            const int k = (launched / kChunk) & 1;
            PG_CUDA(cudaGraphLaunch(exec, s));
            cudaMemcpyAsync(slot[k], m.fl, fl_bytes, cudaMemcpyDeviceToHost, s);
            cudaEventRecord(m.ev[k], s);
            launched += kChunk;
            last = k;
            if (launched > kChunk) {
                PG_CUDA(cudaEventSynchronize(m.ev[1 - k]));
                if (all_done(slot[1 - k])) break;
            }
        }
        PG_CUDA(cudaEventSynchronize(m.ev[last]));
        if (last != 0) std::copy(slot[1], slot[1] + kFlags * m.R, slot[0]);
    }
    return PG_OK;
}

}  // namespace

int mg_build(Ctx& c) {
    if (c.mg) return PG_OK;
    const int rc = build_hierarchy(c);
    if (rc != PG_OK) mg_free(c);
    return rc;
}

void mg_depths(const Ctx& c, std::vector<int>& depth) { depth = c.mg->depth; }

int mg_prepare(Ctx& c, bool f32, bool modes, cudaStream_t s) {
    int rc = mg_build(c);
    if (rc != PG_OK) return rc;
    MgHierarchy& m = *c.mg;
    if ((rc = mg_numeric(c, f32, modes, s))) return rc;
    cudaMemcpyAsync(m.h_fl, m.fl, (size_t)kFlags * m.R * sizeof(int), cudaMemcpyDeviceToHost, s);
    PG_CUDA(cudaStreamSynchronize(s));
    if (m.h_fl[3]) {
        set_error("multigrid: singular coarsest operator");
        return PG_ERR_BREAKDOWN;
    }
    return PG_OK;
}

int mg_precondition(Ctx& c, bool f32, bool modes, cudaStream_t s, const double* r, double* z) {
    MgHierarchy& m = *c.mg;
    if (f32) {
        launch_pdl(k_mg_pre<float>, m.n_cta, kSpanThreads, 0, s, m.spans, c.fixed, r, m.Dinv0f, m.x0f);
        mg_cycle<float>(c, m, modes, s, r, z, nullptr, false);
    } else {
        launch_pdl(k_mg_pre<double>, m.n_cta, kSpanThreads, 0, s, m.spans, c.fixed, r, c.minv, m.x0);
        mg_cycle<double>(c, m, modes, s, r, z, nullptr, false);
    }
    PG_CUDA(cudaGetLastError());
    return PG_OK;
}

void mg_free(Ctx& c) {
    if (!c.mg) return;
    MgHierarchy& m = *c.mg;
    for (cudaGraphExec_t g : m.graph)
        if (g) cudaGraphExecDestroy(g);
    for (cudaEvent_t e : m.ev)
        if (e) cudaEventDestroy(e);
    if (m.h_sc) cudaFreeHost(m.h_sc);
    if (m.h_fl) cudaFreeHost(m.h_fl);
    for (void* p : m.owned) cudaFree(p);
    delete c.mg;
    c.mg = nullptr;
}

int mg_cg(Ctx& c, const pg_solver_cfg& cfg, MgCgResult& res, cudaStream_t s) {
    int rc = mg_build(c);
    if (rc != PG_OK) return rc;
    MgHierarchy& m = *c.mg;
    const bool modes = cfg.inclusion_modes != 0 && m.n_inc > 0;
    rc = cfg.precision == PG_PRECISION_MIXED ? cg_run<float>(c, m, modes, cfg, s) : cg_run<double>(c, m, modes, cfg, s);
    res.scalars = m.h_sc;
    res.flags = m.h_fl;
    return rc;
}

// CG on mask(K) dx = mask(b) (b = c.b, dx = c.dx) preconditioned by one
// V-cycle per iteration.  Fills st.iterations, st.rel_residual (true FP64
// residual) and st.status.
int mg_pcg_solve(Ctx& c, const pg_solver_cfg& cfg, pg_solve_stats& st, cudaStream_t s) {
    MgCgResult res;
    const int rc = mg_cg(c, cfg, res, s);
    if (rc == PG_ERR_BREAKDOWN) {
        st.status = rc;
        return PG_OK;
    }
    if (rc != PG_OK) return rc;
    const double bb = res.scalars[5];
    const double rr = residual_into(c, s, c.dx, c.b, c.r);
    st.iterations = res.flags[2];
    st.refinements = 0;
    st.rel_residual = bb > 0.0 ? std::sqrt(rr / bb) : 0.0;
    if (res.flags[1])
        st.status = PG_ERR_BREAKDOWN;
    else
        st.status = rr <= 4.0 * cfg.rtol * cfg.rtol * bb ? PG_OK : PG_ERR_NOT_CONVERGED;
    return PG_OK;
}

}  // namespace pgb
