// Kernels of the multigrid V-cycle and of the CG around it (see pg_mg.cu).
//
// Every kernel covers all the RVEs of a context (one, or a batch): the work
// is cut into tiles or row spans that lie in one RVE each, listed in a table,
// and a CTA whose RVE is done returns at once.
//
// The kernels are chained by programmatic dependent launch: each starts while
// the one before it runs, reads what no kernel of the chain writes (tables,
// operators, masks, diagonal inverses) and then waits.  Vectors, partial sums,
// scalars and flags are read after the wait only, through loads (lv2, __ldcg)
// that the compiler cannot take for invariant and move ahead of it.
#pragma once

#include "pg_pdl.cuh"
#include "pg_solve_kernels.cuh"

namespace pgb {
namespace mg {

constexpr double kOmegaReg = 0.6;     // level 0, regular nodes: P1 triangles, three nodes each, so
                                      // lambda_max(D^-1 K_rr) <= 3 and 0.6 * 3 < 2
constexpr double kOmega = 0.5;        // coarse levels: four nodes per cell, lambda_max(D^-1 A) <= 4
constexpr int kChebSteps = 4;         // level 0, enrichment nodes
constexpr double kChebRatio = 16.0;   // of the largest to the smallest eigenvalue the polynomial is made for
constexpr int kChebCoef = 8;          // doubles per RVE: 1 / theta, then per later step its two factors
constexpr int kScal = 8;              // doubles per RVE: r.z of even and odd iterations, -, -, tol^2, b.b, true r.r
constexpr int kFlags = 4;             // ints per RVE: done, breakdown, iterations, coarsest operator singular
constexpr int kSpanThreads = 256;
constexpr int kSpanCtasPerSm = 3;     // CTAs of the level-0 kernels that an SM holds: 80 registers, no spills
constexpr int kCoarseCells = 4;       // an RVE is coarsened until both sides have at most this many cells
constexpr int kCoarseMaxDof = 2 * (kCoarseCells + 1) * (kCoarseCells + 1);
constexpr int kCoarseStride = kCoarseMaxDof * kCoarseMaxDof;

// One RVE's grids on the two sides of a transfer: first node and cells per
// side (cnx < 0: the RVE has no such coarse grid).
struct Pair {
    int foff, fnx, fny, coff, cnx, cny;
};

// Row spans of the level-0 kernels: a CTA's RVE and rows, and per RVE its CTAs and where its regular nodes end.
struct Spans {
    const int4* span;       // RVE, first row, end row
    const int2* range;      // per RVE: first CTA, end CTA
    const int* reg_end;     // per RVE
};

// ---------------------------------------------------------------------------
// Grid transfer weights (grid index space).  Coarse index I sits at fine
// index pos(I) = min(2I, nf); nf is the finer grid's cell count.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ int grid_pos(int I, int nf) { return 2 * I < nf ? 2 * I : nf; }

__host__ __device__ __forceinline__ double grid_w(int g, int nf, int I) {
    if ((g & 1) == 0) return (g >> 1) == I ? 1.0 : 0.0;
    if (g == nf) return I == ((nf + 1) >> 1) ? 1.0 : 0.0;
    return (I == ((g - 1) >> 1) || I == ((g + 1) >> 1)) ? 0.5 : 0.0;
}

// The fine indices that restrict to a coarse node at fine index g: g with
// weight 1 and, where g is even, its neighbours with weight 1/2 (an odd g is
// the short last cell's end; its neighbour g - 1 is a coarse node of its own,
// and so is the short cell's other end).
template <typename T>
__device__ __forceinline__ void side_weights(int g, int nf, T& lo, T& hi) {
    lo = (g & 1) == 0 && g > 0 ? (T)0.5 : (T)0;
    hi = (g & 1) == 0 && g + 1 < nf ? (T)0.5 : (T)0;
}

// the two coarse indices a fine index interpolates from, each with weight 1/2 (I0 = I1 where it is only one)
__device__ __forceinline__ void parents(int g, int nf, int& I0, int& I1) {
    I0 = g >> 1;
    I1 = (g + 1) >> 1;
    if (g == nf) I0 = I1;
}

template <typename T>
struct alignas(2 * sizeof(T)) Vec2 {
    T x, y;
};

// a vector's pair (see the head of the file)
__device__ __forceinline__ Vec2<double> lv2(const double* p, size_t i) {
    Vec2<double> v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p + 2 * i));
    return v;
}
__device__ __forceinline__ Vec2<float> lv2(const float* p, size_t i) {
    Vec2<float> v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p + 2 * i));
    return v;
}
template <typename T>
__device__ __forceinline__ void st2(T* p, size_t i, T x, T y) {
    Vec2<T> v;
    v.x = x;
    v.y = y;
    reinterpret_cast<Vec2<T>*>(p)[i] = v;
}

// one 2x2 block of a stencil or a diagonal inverse (volatile: the compiler keeps a row's loads together, ahead
// of the first use, instead of spacing them out to save registers)
__device__ __forceinline__ void load4(const double* p, double& a, double& b, double& c, double& d) {
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p));
}
__device__ __forceinline__ void load4(const float* p, float& a, float& b, float& c, float& d) {
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "l"(p));
}

__device__ __forceinline__ void load2(const double* p, double& a, double& b) {
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "l"(p));
}

// block_sum, valid in every thread
__device__ __forceinline__ double block_sum_all(double v) {
    __shared__ double s_all;
    v = block_sum(v);
    if (threadIdx.x == 0) s_all = v;
    __syncthreads();
    v = s_all;
    __syncthreads();
    return v;
}

// Whether an RVE is done, for every thread of a CTA alike and before its
// kernel's wait, so that no load after the wait stands behind this one (each
// kernel of the chain had a trip to memory more: 512^2 FP64 8.96 -> 8.06 ms,
// the cohesive 256^2 path 162 -> 140).  The flag may be set
// meanwhile: a kernel that misses that forms vectors nobody reads, as x and
// the iteration count change in k_cg_update alone, which looks after its wait.
__device__ __forceinline__ bool cta_done(const int* fl, int r) {
    return fl && __syncthreads_or(__ldcg(&fl[kFlags * r]));
}

// The sum of one RVE's partials, in CTA order.  A reduction's kernel leaves
// one partial per CTA and the next kernel's CTAs each add them up: the kernel
// boundary orders the two, so no CTA waits on a fence and a ticket (which held
// every CTA of the earlier fused sums: 33 us against 21 us for the same matrix
// product without a sum at 512^2), and the result is the same bits on every run.
__device__ __forceinline__ double range_sum(const double* part, int2 rg) {
    double v = 0.0;
    for (int k = rg.x + threadIdx.x; k < rg.y; k += blockDim.x) v += __ldcg(&part[k]);
    return block_sum_all(v);
}

// Block rows of K times a vector, kRowLanes lanes per row: lane g takes the
// row's blocks g, g + kRowLanes, ... (a group's loads of K are contiguous).
// RowFrag holds the columns and blocks of a lane's first kRowUnroll of them
// (rows of up to 12 blocks), issued together; the first rows' are loaded
// before the kernel's wait.
template <typename MT>
struct RowFrag {
    int r1, next;              // end of the row, and the lane's first block beyond the fragment
    int j[kRowUnroll];
    MT b[kRowUnroll][4];

    __device__ __forceinline__ void blocks(int base, const int* __restrict__ col, const MT* __restrict__ K) {
#pragma unroll
        for (int u = 0; u < kRowUnroll; ++u) {
            const int k = base + u * kRowLanes;
            j[u] = -1;
            if (k < r1) {
                j[u] = __ldg(&col[k]);
                load4(K + 4 * (size_t)k, b[u][0], b[u][1], b[u][2], b[u][3]);
            }
        }
        next = base + kRowUnroll * kRowLanes;
    }
    __device__ __forceinline__ void load(int i, bool valid, int g, const int* __restrict__ row_ptr,
                                         const int* __restrict__ col, const MT* __restrict__ K) {
        const int r0 = valid ? __ldg(&row_ptr[i]) : 0;
        r1 = valid ? __ldg(&row_ptr[i + 1]) : 0;
        blocks(r0 + g, col, K);
    }
    // the row's product, in every lane of its group; get(j) is the vector's pair at column node j
    template <typename Get>
    __device__ __forceinline__ void dot(const int* __restrict__ col, const MT* __restrict__ K, Get get, double& y0,
                                        double& y1) {
        double a0 = 0.0, a1 = 0.0;
        while (true) {
            Vec2<double> v[kRowUnroll];
#pragma unroll
            for (int u = 0; u < kRowUnroll; ++u)
                if (j[u] >= 0) v[u] = get(j[u]);
#pragma unroll
            for (int u = 0; u < kRowUnroll; ++u)
                if (j[u] >= 0) {
                    a0 += (double)b[u][0] * v[u].x + (double)b[u][1] * v[u].y;
                    a1 += (double)b[u][2] * v[u].x + (double)b[u][3] * v[u].y;
                }
            if (next >= r1) break;
            blocks(next, col, K);
        }
        a0 += __shfl_xor_sync(0xffffffffu, a0, 1);
        a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
        a0 += __shfl_xor_sync(0xffffffffu, a0, 2);
        a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
        y0 = a0;
        y1 = a1;
    }
};
// Block rows i0 .. i0 + n (n <= 32) of K times a vector, one warp: lane l
// returns row i0 + l.  The lanes take the rows' blocks in storage order, U at
// a time (a warp's loads of K are whole lines, and no lane waits for a longer
// row's), leave each block's product in shared memory (sp, kWarpBlocks
// entries of the warp's own) and then each sums its row there, in order.
// For the level-0 products, which four lanes per row read with half the lanes
// of a last round idle: K p of 512^2 26.6 -> 20.5 us, of 1000 x 700 68 -> 60
// (bound by the latency of its trips to memory -- row, blocks and columns,
// vector -- at 24 warps per SM; K alone takes 24 at the DRAM's rate).  More
// warps with fewer blocks in flight, chunks of K copied ahead with cp.async,
// and K kept in an order without column indices were all slower.
constexpr int kWarpBlocks = 256;
template <int U, typename MT, typename Get>
__device__ __forceinline__ void warp_rows(int i0, int n, const int* __restrict__ row_ptr, const int* __restrict__ col,
                                          const MT* __restrict__ K, Get get, double2* sp, double& y0, double& y1) {
    const int lane = threadIdx.x & 31;
    const int r0 = __ldg(&row_ptr[i0 + min(lane, n)]), r1 = __ldg(&row_ptr[i0 + min(lane + 1, n)]);
    const int begin = __shfl_sync(0xffffffffu, r0, 0), end = __shfl_sync(0xffffffffu, r1, 31);
    y0 = y1 = 0.0;
    for (int c0 = begin; c0 < end; c0 += kWarpBlocks) {
        const int c1 = min(end, c0 + kWarpBlocks);
        for (int base = c0 + lane; base < c1; base += 32 * U) {
            int j[U];
            MT b[U][4];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = base + 32 * u;
                j[u] = -1;
                if (k < c1) {
                    j[u] = __ldg(&col[k]);
                    load4(K + 4 * (size_t)k, b[u][0], b[u][1], b[u][2], b[u][3]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (j[u] >= 0) {
                    const Vec2<double> v = get(j[u]);
                    sp[base + 32 * u - c0] = make_double2((double)b[u][0] * v.x + (double)b[u][1] * v.y,
                                                          (double)b[u][2] * v.x + (double)b[u][3] * v.y);
                }
            }
        }
        __syncwarp();
        const int k1 = min(r1, c1);
        for (int k = max(r0, c0); k < k1; ++k) {
            y0 += sp[k - c0].x;
            y1 += sp[k - c0].y;
        }
        __syncwarp();
    }
}
// the part of a CTA's rows that a warp takes, and how many of them at once
struct WarpSpan {
    int i, end, step;
};
__device__ __forceinline__ WarpSpan warp_span(int begin, int end) {
    const int w = threadIdx.x >> 5, n = max(0, end - begin);
    WarpSpan s;
    s.i = begin + (int)((long long)n * w / (kSpanThreads / 32));
    s.end = begin + (int)((long long)n * (w + 1) / (kSpanThreads / 32));
    const int parts = (s.end - s.i + 31) / 32;
    s.step = parts > 0 ? (s.end - s.i + parts - 1) / parts : 32;
    return s;
}
template <typename T>
__device__ __forceinline__ Vec2<double> widen(Vec2<T> a) {
    Vec2<double> v;
    v.x = (double)a.x;
    v.y = (double)a.y;
    return v;
}

// ---------------------------------------------------------------------------
// CG.  Iteration parity P; part_* hold one partial per CTA of the spans.
// ---------------------------------------------------------------------------

// x = 0, r = mask(b); partials of r.r; the first regular smoothing sweep x1 = omega D^-1 r
template <typename T>
__global__ void __launch_bounds__(kSpanThreads) k_cg_start(Spans sp, const uint8_t* __restrict__ fixed, const double* b,
                                                           double* r, double* x, const T* Dinv, T* x1, double* part_rr) {
    pdl_wait();
    pdl_trigger();
    const int4 S = sp.span[blockIdx.x];
    const int reg = sp.reg_end[S.x];
    double acc = 0.0;
    for (int i = S.y + threadIdx.x; i < S.z; i += kSpanThreads) {
        const Vec2<double> v = lv2(b, i);
        const double r0 = fixed[2 * i] ? 0.0 : v.x, r1 = fixed[2 * i + 1] ? 0.0 : v.y;
        st2(r, i, r0, r1);
        st2(x, i, 0.0, 0.0);
        acc += r0 * r0 + r1 * r1;
        if (i < reg) {
            T m0, m1, m2, m3;
            load4(Dinv + 4 * (size_t)i, m0, m1, m2, m3);
            st2(x1, i, (T)kOmegaReg * (m0 * (T)r0 + m1 * (T)r1), (T)kOmegaReg * (m2 * (T)r0 + m3 * (T)r1));
        }
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part_rr[blockIdx.x] = acc;
}

// the first regular smoothing sweep alone (a V-cycle applied outside CG)
template <typename T>
__global__ void __launch_bounds__(kSpanThreads) k_mg_pre(Spans sp, const uint8_t* __restrict__ fixed, const double* r,
                                                         const T* Dinv, T* x1) {
    pdl_wait();
    pdl_trigger();
    const int4 S = sp.span[blockIdx.x];
    const int end = min(S.z, sp.reg_end[S.x]);
    for (int i = S.y + threadIdx.x; i < end; i += kSpanThreads) {
        const Vec2<double> v = lv2(r, i);
        const T r0 = fixed[2 * i] ? (T)0 : (T)v.x, r1 = fixed[2 * i + 1] ? (T)0 : (T)v.y;
        T m0, m1, m2, m3;
        load4(Dinv + 4 * (size_t)i, m0, m1, m2, m3);
        st2(x1, i, (T)kOmegaReg * (m0 * r0 + m1 * r1), (T)kOmegaReg * (m2 * r0 + m3 * r1));
    }
}

// per RVE: tol^2 = rtol^2 b.b, and the r.z that the first iteration divides by
__global__ inline void k_cg_tol(Spans sp, const double* part_rr, double rtol2, double* sc, int* fl) {
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.x;
    const double bb = range_sum(part_rr, sp.range[r]);
    if (threadIdx.x == 0) {
        double* s = sc + kScal * r;
        s[0] = 0.0;
        s[1] = 1.0;
        s[4] = rtol2 * bb;
        s[5] = bb;
        if (bb == 0.0) fl[kFlags * r] = 1;
    }
}

// p = z + beta p_old, q = mask(K p), partials of p.q.  p is formed where it is
// read: a row gathers z and p_old of its columns instead of waiting for a
// kernel that writes p.  Bound by the reads of K (32 bytes a block).
__global__ void __launch_bounds__(kSpanThreads, kSpanCtasPerSm) k_cg_spmv(Spans sp, const int* __restrict__ row_ptr,
                                                          const int* __restrict__ col, const double* __restrict__ K,
                                                          const uint8_t* __restrict__ fixed, const double* z,
                                                          const double* p_old, double* p, double* q, const double* part_rz,
                                                          double* sc, const int* fl, double* part_pq, int P) {
    __shared__ double2 s_rows[kSpanThreads / 32 * kWarpBlocks];
    const int4 S = sp.span[blockIdx.x];
    const int2 rg = sp.range[S.x];
    const bool done = cta_done(fl, S.x);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    double* s = sc + kScal * S.x;
    const double rz_old = __ldcg(&s[1 - P]);
    const double rz = range_sum(part_rz, rg);
    const double beta = rz / rz_old;
    if ((int)blockIdx.x == rg.x && threadIdx.x == 0) s[P] = rz;
    double acc = 0.0;
    for (WarpSpan ws = warp_span(S.y, S.z); ws.i < ws.end; ws.i += ws.step) {
        const int n = min(ws.step, ws.end - ws.i), i = ws.i + (threadIdx.x & 31);
        double y0, y1;
        warp_rows<4>(ws.i, n, row_ptr, col, K, [&](int j) {
            Vec2<double> a = lv2(z, j);
            const Vec2<double> b = lv2(p_old, j);
            a.x += beta * b.x;
            a.y += beta * b.y;
            return a;
        }, s_rows + kWarpBlocks * (threadIdx.x >> 5), y0, y1);
        if (i < ws.i + n) {
            const Vec2<double> a = lv2(z, i), b = lv2(p_old, i);
            const double p0 = a.x + beta * b.x, p1 = a.y + beta * b.y;
            if (fixed[2 * i]) y0 = 0.0;
            if (fixed[2 * i + 1]) y1 = 0.0;
            st2(p, i, p0, p1);
            st2(q, i, y0, y1);
            acc += p0 * y0 + p1 * y1;
        }
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part_pq[blockIdx.x] = acc;
}

// x += alpha p, r -= alpha q, partials of r.r, and the first regular smoothing sweep of the coming V-cycle
template <typename T>
__global__ void __launch_bounds__(kSpanThreads) k_cg_update(Spans sp, double* x, double* r, const double* p, const double* q,
                                                            const T* __restrict__ Dinv, T* x1, const double* part_pq,
                                                            const double* sc, int* fl, double* part_rr, int P) {
    const int4 S = sp.span[blockIdx.x];
    const int2 rg = sp.range[S.x];
    const int reg = sp.reg_end[S.x];
    const bool was_done = cta_done(fl, S.x);
    pdl_wait();
    pdl_trigger();
    if (was_done) return;
    int* f = fl + kFlags * S.x;
    const int done = __ldcg(&f[0]);
    // a thread's first vectors are on their way while alpha is summed (a small system's CTA has one node per thread)
    int i = S.y + threadIdx.x;
    Vec2<double> xv, rv, pv, qv;
    auto load = [&] {
        if (i >= S.z) return;
        xv = lv2(x, i);
        rv = lv2(r, i);
        pv = lv2(p, i);
        qv = lv2(q, i);
    };
    load();
    const double rz = __ldcg(&sc[kScal * S.x + P]);
    const double pq = range_sum(part_pq, rg);
    if (done) return;
    const bool first = (int)blockIdx.x == rg.x && threadIdx.x == 0;
    if (!(pq > 0.0)) {
        if (first) {
            f[1] = 1;
            f[0] = 1;
        }
        return;
    }
    if (first) f[2] += 1;
    const double alpha = rz / pq;
    double acc = 0.0;
    while (i < S.z) {
        const double r0 = rv.x - alpha * qv.x, r1 = rv.y - alpha * qv.y;
        st2(x, i, xv.x + alpha * pv.x, xv.y + alpha * pv.y);
        st2(r, i, r0, r1);
        acc += r0 * r0 + r1 * r1;
        if (i < reg) {
            T m0, m1, m2, m3;
            load4(Dinv + 4 * (size_t)i, m0, m1, m2, m3);
            st2(x1, i, (T)kOmegaReg * (m0 * (T)r0 + m1 * (T)r1), (T)kOmegaReg * (m2 * (T)r0 + m3 * (T)r1));
        }
        i += kSpanThreads;
        load();
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part_rr[blockIdx.x] = acc;
}

// partials of a.b
__global__ inline void __launch_bounds__(kSpanThreads) k_cg_dot(Spans sp, const double* a, const double* b, const int* fl,
                                                                double* part) {
    const int4 S = sp.span[blockIdx.x];
    const bool done = cta_done(fl, S.x);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    double acc = 0.0;
    for (int i = S.y + threadIdx.x; i < S.z; i += kSpanThreads) {
        const Vec2<double> u = lv2(a, i), v = lv2(b, i);
        acc += u.x * v.x + u.y * v.y;
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// ---------------------------------------------------------------------------
// Level 0
// ---------------------------------------------------------------------------

// The enrichment nodes' part of the smoother: x_e (+)= q(D^-1 K_ee) D^-1 r_e
// with the Chebyshev polynomial q of degree kChebSteps - 1 for the spectrum
// (bound / kChebRatio, bound), r_e the residual at x.  The enrichment block
// couples each interface's nodes along a chain; damped block Jacobi sweeps of
// the whole system resolve it slowly (72 CG iterations at 128^2, 154 with
// softened cohesive interfaces; 53 and 84 with one regular sweep and this).
//
// A piece is up to kPieceRows enrichment nodes and those around it that its
// steps need: step k reads the previous iterate one node further out, so the
// nodes within kChebSteps - 1 - k steps are recomputed and the piece needs no
// exchange with others (the result is the polynomial of the whole K_ee).
// Four lanes per row; one latency chain per step is what bounds it.
struct Piece {
    int row0;                  // its first local row; then rows at distance 0, <= 1, <= 2, <= 3
    int end[kChebSteps];
    int rve, pad0, pad1;
};
constexpr int kPieceRows = 48;
// Threads per CTA: all of a piece's rows at once, as a row beyond the first
// TH / kRowLanes loads its numbers and blocks again in every step (pieces of
// 60 to 108 rows, 256^2 cohesive, FP32: 9.3 us with 256 threads, 8.4 with 448).
constexpr int kPieceThreads = 256, kPieceThreadsWide = 448;

struct Enr {
    const Piece* piece;
    const int* node;           // per local row: its node
    const int* eptr;           // per local row: its entries in K_ee
    const int2* ent;           // block slot in K, local column
    const double* coef;        // kChebCoef per RVE
};

template <typename T, bool POST, int TH>
__global__ void __launch_bounds__(TH, TH == kPieceThreads ? 3 : 2) k_mg_enr(Enr e, const int* __restrict__ row_ptr, const int* __restrict__ col,
                                                          const T* __restrict__ K, const T* __restrict__ Dinv,
                                                          const uint8_t* __restrict__ fixed, const int* __restrict__ reg_end,
                                                          const double* b, const T* xin, T* xout, const int* fl) {
    extern __shared__ __align__(16) unsigned char enr_smem[];
    const Piece pc = e.piece[blockIdx.x];
    const int n = pc.end[kChebSteps - 1];
    Vec2<T>* sx = reinterpret_cast<Vec2<T>*>(enr_smem);  // two copies of x, then d and r
    Vec2<T>* sx2 = sx + n;
    Vec2<T>* sd = sx2 + n;
    Vec2<T>* sr = sd + n;
    const double* cf = e.coef + kChebCoef * pc.rve;
    const int reg = reg_end[pc.rve];
    const int g = threadIdx.x % kRowLanes, l0 = threadIdx.x / kRowLanes;
    constexpr int kRows = TH / kRowLanes;
    constexpr int kEnt = 2;  // entries of K_ee that a lane keeps of its row among the first kRows (8 a row)
    int i = l0 < n ? e.node[pc.row0 + l0] : 0;
    RowFrag<T> f;
    f.load(i, l0 < n, g, row_ptr, col, K);
    const int e0 = l0 < n ? e.eptr[pc.row0 + l0] : 0, e1 = l0 < n ? e.eptr[pc.row0 + l0 + 1] : 0;
    int ec[kEnt];
    T eb[kEnt][4];
#pragma unroll
    for (int u = 0; u < kEnt; ++u) {
        const int q = e0 + g + u * kRowLanes;
        ec[u] = -1;
        if (q < e1) {
            const int2 en = __ldg(&e.ent[q]);
            ec[u] = en.y;
            load4(K + 4 * (size_t)en.x, eb[u][0], eb[u][1], eb[u][2], eb[u][3]);
        }
    }
    T m0, m1, m2, m3;  // of the row among the first kRows
    load4(Dinv + 4 * (size_t)i, m0, m1, m2, m3);
    const bool f0 = fixed[2 * i], f1 = fixed[2 * i + 1];
    T c[2 * kChebSteps - 1];
#pragma unroll
    for (int k = 0; k < 2 * kChebSteps - 1; ++k) c[k] = (T)cf[k];
    const bool done = cta_done(fl, pc.rve);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    for (int base = 0; base < n; base += kRows) {
        const int l = base + l0;
        if (base > 0) {
            i = l < n ? e.node[pc.row0 + l] : 0;
            f.load(i, l < n, g, row_ptr, col, K);
        }
        const Vec2<double> bv = lv2(b, i);
        double y0, y1;
        f.dot(col, K, [&](int j) {
            Vec2<double> v;
            v.x = v.y = 0.0;
            if (POST || j < reg) v = widen(lv2(xin, j));  // before the coarse correction x_e is zero
            return v;
        }, y0, y1);
        if (l < n && g == 0) {
            Vec2<T> rv, dv;
            T a0 = m0, a1 = m1, a2 = m2, a3 = m3;
            if (base > 0) load4(Dinv + 4 * (size_t)i, a0, a1, a2, a3);
            rv.x = fixed[2 * i] ? (T)0 : (T)bv.x - (T)y0;
            rv.y = fixed[2 * i + 1] ? (T)0 : (T)bv.y - (T)y1;
            dv.x = c[0] * (a0 * rv.x + a1 * rv.y);
            dv.y = c[0] * (a2 * rv.x + a3 * rv.y);
            sr[l] = rv;
            sd[l] = dv;
            sx[l] = dv;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 1; k < kChebSteps; ++k) {
        const T c1 = c[2 * k - 1], c2 = c[2 * k];
        const int rows = pc.end[kChebSteps - 1 - k];
        const Vec2<T>* xa = (k & 1) ? sx : sx2;
        Vec2<T>* xb = (k & 1) ? sx2 : sx;
        for (int base = 0; base < rows; base += kRows) {
            const int l = base + l0;
            double a0 = 0.0, a1 = 0.0;
            int q = e0 + g, q1 = e1;
            if (base == 0) {
#pragma unroll
                for (int u = 0; u < kEnt; ++u)
                    if (ec[u] >= 0) {
                        const Vec2<T> v = xa[ec[u]];
                        a0 += (double)eb[u][0] * (double)v.x + (double)eb[u][1] * (double)v.y;
                        a1 += (double)eb[u][2] * (double)v.x + (double)eb[u][3] * (double)v.y;
                    }
                q += kEnt * kRowLanes;
            } else {
                q = l < rows ? e.eptr[pc.row0 + l] + g : 0;
                q1 = l < rows ? e.eptr[pc.row0 + l + 1] : 0;
            }
            for (; q < q1; q += kRowLanes) {
                const int2 en = __ldg(&e.ent[q]);
                double k0, k1, k2, k3;
                load_block(K + 4 * (size_t)en.x, k0, k1, k2, k3);
                const Vec2<T> v = xa[en.y];
                a0 += k0 * (double)v.x + k1 * (double)v.y;
                a1 += k2 * (double)v.x + k3 * (double)v.y;
            }
            a0 += __shfl_xor_sync(0xffffffffu, a0, 1);
            a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
            a0 += __shfl_xor_sync(0xffffffffu, a0, 2);
            a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
            if (l < rows && g == 0) {
                T n0 = m0, n1 = m1, n2 = m2, n3 = m3;
                bool g0 = f0, g1 = f1;
                if (base > 0) {
                    const int il = e.node[pc.row0 + l];
                    load4(Dinv + 4 * (size_t)il, n0, n1, n2, n3);
                    g0 = fixed[2 * il];
                    g1 = fixed[2 * il + 1];
                }
                const T r0 = g0 ? (T)0 : sr[l].x - (T)a0, r1 = g1 ? (T)0 : sr[l].y - (T)a1;
                Vec2<T> dv = sd[l], xv = xa[l];
                dv.x = c1 * dv.x + c2 * (n0 * r0 + n1 * r1);
                dv.y = c1 * dv.y + c2 * (n2 * r0 + n3 * r1);
                xv.x += dv.x;
                xv.y += dv.y;
                sd[l] = dv;
                xb[l] = xv;
            }
        }
        __syncthreads();
    }
    const Vec2<T>* xl = ((kChebSteps - 1) & 1) ? sx2 : sx;
    for (int l = threadIdx.x; l < pc.end[0]; l += TH) {
        const int il = e.node[pc.row0 + l];
        Vec2<T> v = xl[l];
        if (POST) {
            const Vec2<T> o = lv2(xin, il);
            v.x += o.x;
            v.y += o.y;
        }
        st2(xout, il, v.x, v.y);
    }
}

// Level-0 residual at the regular nodes of a tile of coarse nodes, restricted
// to them: b_1 = mask(P^T (b - K x)).  Tiles of 8 x 8 coarse nodes need the
// residual of 17 x 17 fine ones (13% computed twice), which saves writing it
// and a launch.  The tile marked first in its RVE also ends the CG iteration:
// it sets the RVE's done flag when the update's r.r has reached the tolerance.
constexpr int kDownTile = 8;
constexpr int kDownFine = 2 * kDownTile + 1;

template <typename T>
__device__ __forceinline__ void restrict_tile(const Vec2<T>* s, int I0, int J0, const Pair& p,
                                              const uint8_t* __restrict__ fixed_c, T* bc) {
    // s: the residual on fine nodes (2 I0 - 1 .., 2 J0 - 1 ..), kDownFine per side, 0 outside the grid
    const int t = threadIdx.x;
    if (t >= kDownTile * kDownTile) return;
    const int I = I0 + t % kDownTile, J = J0 + t / kDownTile;
    if (I > p.cnx || J > p.cny) return;
    const int gx = grid_pos(I, p.fnx), gy = grid_pos(J, p.fny);
    T wx[3], wy[3];
    side_weights(gx, p.fnx, wx[0], wx[2]);
    side_weights(gy, p.fny, wy[0], wy[2]);
    wx[1] = wy[1] = (T)1;
    const Vec2<T>* c = s + (gy - (2 * J0 - 1)) * kDownFine + gx - (2 * I0 - 1);
    T s0 = 0, s1 = 0;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const T w = wy[dy + 1] * wx[dx + 1];
            if (w == (T)0) continue;
            const Vec2<T> v = c[dy * kDownFine + dx];
            s0 += w * v.x;
            s1 += w * v.y;
        }
    const int a = p.coff + I + J * (p.cnx + 1);
    st2(bc, a, fixed_c[2 * a] ? (T)0 : s0, fixed_c[2 * a + 1] ? (T)0 : s1);
}

// 9 warps take the tile's 17 rows of 17 nodes in two rounds.
constexpr int kDown0Threads = 288;
template <typename T>
__global__ void __launch_bounds__(kDown0Threads, sizeof(T) == 8 ? 4 : 3) k_mg_down0(const int4* __restrict__ tile, const Pair* __restrict__ pair,
                                                            const int* __restrict__ row_ptr, const int* __restrict__ col,
                                                            const T* __restrict__ K, const uint8_t* __restrict__ fixed,
                                                            const double* b, const T* x, const uint8_t* __restrict__ fixed_c,
                                                            T* bc, Spans sp, const double* part_rr, const double* sc,
                                                            int* fl, int check) {
    __shared__ Vec2<T> s[kDownFine * kDownFine];
    __shared__ double2 s_rows[kDown0Threads / 32 * kWarpBlocks];
    const int4 tl = tile[blockIdx.x];
    const Pair p = pair[tl.x];
    const int gx0 = 2 * tl.y - 1, gy0 = 2 * tl.z - 1;
    const bool done = cta_done(fl, tl.x);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    if (check && tl.w) {
        const double rr = range_sum(part_rr, sp.range[tl.x]);
        if (threadIdx.x == 0 && rr <= __ldcg(&sc[kScal * tl.x + 4])) fl[kFlags * tl.x] = 1;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gxa = max(gx0, 0), n = min(gx0 + kDownFine - 1, p.fnx) + 1 - gxa;  // the tile's columns inside the grid
    for (int ly = w; ly < kDownFine; ly += kDown0Threads / 32) {
        const int gy = gy0 + ly, i0 = p.foff + gxa + gy * (p.fnx + 1);
        Vec2<T> rv;
        rv.x = rv.y = 0;
        if (gy >= 0 && gy <= p.fny) {
            double y0, y1;
            warp_rows<sizeof(T) == 8 ? 2 : 4>(i0, n, row_ptr, col, K, [&](int j) { return widen(lv2(x, j)); },
                                              s_rows + kWarpBlocks * w, y0, y1);
            if (lane < n) {
                const int i = i0 + lane;
                const Vec2<double> bv = lv2(b, i);
                rv.x = fixed[2 * i] ? (T)0 : (T)bv.x - (T)y0;
                rv.y = fixed[2 * i + 1] ? (T)0 : (T)bv.y - (T)y1;
            }
        }
        // lanes beyond the grid's columns clear the tile's others
        const int lx = lane < n ? lane + gxa - gx0 : lane - n < gxa - gx0 ? lane - n : lane;
        if (lx < kDownFine) s[ly * kDownFine + lx] = rv;
    }
    __syncthreads();
    restrict_tile(s, tl.y, tl.z, p, fixed_c, bc);
}

// The last smoothing sweep (regular nodes) and z: z_r = x_r + omega D^-1 (b - K x), z_e = x_e (already
// smoothed, in xe); partials of b.z, which CG takes as r.z
template <typename T>
__global__ void __launch_bounds__(kSpanThreads, kSpanCtasPerSm) k_mg_post(Spans sp, const int* __restrict__ row_ptr,
                                                          const int* __restrict__ col, const T* __restrict__ K,
                                                          const T* __restrict__ Dinv, const uint8_t* __restrict__ fixed,
                                                          const double* b, const T* x, const T* xe, double* z, const int* fl,
                                                          double* part_rz) {
    __shared__ double2 s_rows[kSpanThreads / 32 * kWarpBlocks];
    const int4 S = sp.span[blockIdx.x];
    const int reg = sp.reg_end[S.x];
    const bool done = cta_done(fl, S.x);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    double acc = 0.0;
    for (WarpSpan ws = warp_span(S.y, min(S.z, reg)); ws.i < ws.end; ws.i += ws.step) {
        const int n = min(ws.step, ws.end - ws.i), i = ws.i + (threadIdx.x & 31);
        double y0, y1;
        Vec2<double> bv;
        Vec2<T> xv;
        T m0, m1, m2, m3;
        uchar2 fx;
        if (i < ws.i + n) {
            bv = lv2(b, i);
            xv = lv2(x, i);
            fx = __ldg(reinterpret_cast<const uchar2*>(fixed) + i);
            load4(Dinv + 4 * (size_t)i, m0, m1, m2, m3);
        }
        warp_rows<4>(ws.i, n, row_ptr, col, K, [&](int j) { return widen(lv2(j < reg ? x : xe, j)); },
                     s_rows + kWarpBlocks * (threadIdx.x >> 5), y0, y1);
        if (i < ws.i + n) {
            const T t0 = fx.x ? (T)0 : (T)bv.x - (T)y0, t1 = fx.y ? (T)0 : (T)bv.y - (T)y1;
            const double z0 = (double)(xv.x + (T)kOmegaReg * (m0 * t0 + m1 * t1));
            const double z1 = (double)(xv.y + (T)kOmegaReg * (m2 * t0 + m3 * t1));
            st2(z, i, z0, z1);
            acc += bv.x * z0 + bv.y * z1;
        }
    }
    for (int k = max(S.y, reg) + threadIdx.x; k < S.z; k += kSpanThreads) {
        const Vec2<double> bv = lv2(b, k), xv = widen(lv2(xe, k));
        st2(z, k, xv.x, xv.y);
        acc += bv.x * xv.x + bv.y * xv.y;
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) part_rz[blockIdx.x] = acc;
}

// ---------------------------------------------------------------------------
// Coarse levels: 9-point block stencils, two sweeps of damped block Jacobi
// each way.  One launch per level and direction: a launch on these levels
// costs 3-5 us whatever its size, and a level took seven.  A CTA recomputes
// the nodes around its tile that the next phase reads (27% more sweeps)
// instead of waiting for its neighbours.
// ---------------------------------------------------------------------------
//
// A thread keeps one node of the tile's first swept region through all the
// phases, so its operator row is loaded once, before the wait.  448 threads:
// the 441 nodes that the first sweep reads are staged in one round of loads
// (384 threads took two: 3% of a 256^2 solve in FP64, 1.5% of 512^2).
constexpr int kTileThreads = 448;

template <typename T>
struct NodeRow {
    T k[9][4], m[4];
    __device__ __forceinline__ void load(int i, const T* __restrict__ A, const T* __restrict__ Dinv) {
#pragma unroll
        for (int q = 0; q < 9; ++q) load4(A + 36 * (size_t)i + 4 * q, k[q][0], k[q][1], k[q][2], k[q][3]);
        load4(Dinv + 4 * (size_t)i, m[0], m[1], m[2], m[3]);
    }
    // b - A x from x staged in shared memory, at s[l] of a region W wide (0 at a fixed DOF: its row and b are)
    __device__ __forceinline__ Vec2<T> residual(Vec2<T> b, const Vec2<T>* s, int l, int W) const {
        T y0 = 0, y1 = 0;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const Vec2<T> v = s[l + (q / 3 - 1) * W + q % 3 - 1];
            y0 += k[q][0] * v.x + k[q][1] * v.y;
            y1 += k[q][2] * v.x + k[q][3] * v.y;
        }
        b.x -= y0;
        b.y -= y1;
        return b;
    }
    // x + omega D^-1 r
    __device__ __forceinline__ Vec2<T> relax(Vec2<T> x, Vec2<T> r) const {
        x.x += (T)kOmega * (m[0] * r.x + m[1] * r.y);
        x.y += (T)kOmega * (m[2] * r.x + m[3] * r.y);
        return x;
    }
};

// pre-smoothing from zero, residual, restriction: x of the finer grid's nodes and b of the coarser one's
template <typename T>
__global__ void __launch_bounds__(kTileThreads, sizeof(T) == 8 ? 1 : 2) k_mg_down(const int4* __restrict__ tile,
                                                                                  const Pair* __restrict__ pair,
                                                                                  const T* __restrict__ A,
                                                                                  const T* __restrict__ Dinv, const T* b, T* x,
                                                                                  const uint8_t* __restrict__ fixed_c, T* bc,
                                                                                  const int* fl) {
    constexpr int W0 = kDownFine, W1 = W0 + 2, W2 = W1 + 2;
    static_assert(W1 * W1 <= kTileThreads, "one thread per node of the swept region");
    __shared__ Vec2<T> s1[W2 * W2];  // after one sweep
    __shared__ Vec2<T> s2[W1 * W1];  // after two
    __shared__ Vec2<T> s0[W0 * W0];  // residual
    const int4 tl = tile[blockIdx.x];
    const Pair p = pair[tl.x];
    const int gx0 = 2 * tl.y - 2, gy0 = 2 * tl.z - 2;  // of the swept region
    const int t = threadIdx.x, lx = t % W1, ly = t / W1, gx = gx0 + lx, gy = gy0 + ly;
    const bool in = t < W1 * W1 && gx >= 0 && gx <= p.fnx && gy >= 0 && gy <= p.fny;
    const int i = in ? p.foff + gx + gy * (p.fnx + 1) : p.foff;
    NodeRow<T> row;
    row.load(i, A, Dinv);
    const bool done = cta_done(fl, tl.x);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    Vec2<T> bv = lv2(b, i);
    for (int l = t; l < W2 * W2; l += kTileThreads) {
        const int hx = gx0 - 1 + l % W2, hy = gy0 - 1 + l / W2;
        Vec2<T> v;
        v.x = v.y = 0;
        if (hx >= 0 && hx <= p.fnx && hy >= 0 && hy <= p.fny) {
            const int h = p.foff + hx + hy * (p.fnx + 1);
            const Vec2<T> r = lv2(b, h);  // (masked by the restriction)
            T m0, m1, m2, m3;
            load4(Dinv + 4 * (size_t)h, m0, m1, m2, m3);
            v.x = (T)kOmega * (m0 * r.x + m1 * r.y);
            v.y = (T)kOmega * (m2 * r.x + m3 * r.y);
        }
        s1[l] = v;
    }
    __syncthreads();
    const int c = (ly + 1) * W2 + lx + 1;
    if (t < W1 * W1) {
        Vec2<T> v;
        v.x = v.y = 0;
        if (in) {
            v = row.relax(s1[c], row.residual(bv, s1, c, W2));
            // a fine node belongs to the tile of its index / (2 kDownTile)
            if (gx >= 2 * tl.y && gx < 2 * (tl.y + kDownTile) && gy >= 2 * tl.z && gy < 2 * (tl.z + kDownTile))
                st2(x, i, v.x, v.y);
        }
        s2[t] = v;
    }
    __syncthreads();
    if (lx >= 1 && lx <= W0 && ly >= 1 && ly <= W0) {
        Vec2<T> v;
        v.x = v.y = 0;
        if (in) v = row.residual(bv, s2, t, W1);
        s0[(ly - 1) * W0 + lx - 1] = v;
    }
    __syncthreads();
    restrict_tile(s0, tl.y, tl.z, p, fixed_c, bc);
}

// the coarse correction at fine node (gx, gy)
template <typename T>
__device__ __forceinline__ Vec2<T> interpolate(int gx, int gy, const Pair& p, const T* xc) {
    int I0, I1, J0, J1;
    parents(gx, p.fnx, I0, I1);
    parents(gy, p.fny, J0, J1);
    const int W = p.cnx + 1;
    const Vec2<T> a = lv2(xc, p.coff + I0 + J0 * W), b = lv2(xc, p.coff + I1 + J0 * W);
    const Vec2<T> c = lv2(xc, p.coff + I0 + J1 * W), d = lv2(xc, p.coff + I1 + J1 * W);
    Vec2<T> v;
    v.x = (T)0.25 * ((a.x + b.x) + (c.x + d.x));
    v.y = (T)0.25 * ((a.y + b.y) + (c.y + d.y));
    return v;
}

// Coarse correction and post-smoothing of one level (the coarse side of
// `pair`, the fine side of `pairc`).  FINE: its result is interpolated
// straight into level 0's x; otherwise it goes to xo.
constexpr int kUpTile = 16;
template <typename T, bool FINE>
__global__ void __launch_bounds__(kTileThreads, sizeof(T) == 8 ? 1 : 2) k_mg_up(const int4* __restrict__ tile, const Pair* __restrict__ pair,
                                                           const Pair* __restrict__ pairc, const T* __restrict__ A,
                                                           const T* __restrict__ Dinv, const uint8_t* __restrict__ fixed,
                                                           const T* b, const T* x, const T* xc, T* xo,
                                                           const uint8_t* __restrict__ fixed0, T* x0, const int* fl) {
    constexpr int W0 = kUpTile + (FINE ? 1 : 0), W1 = W0 + 2, W2 = W1 + 2;
    static_assert(W1 * W1 <= kTileThreads, "one thread per node of the swept region");
    __shared__ Vec2<T> s2[W2 * W2];  // corrected
    __shared__ Vec2<T> s1[W1 * W1];  // after one sweep
    __shared__ Vec2<T> s0[W0 * W0];  // after two
    const int4 tl = tile[blockIdx.x];
    const Pair pf = pair[tl.x], p = pairc[tl.x];
    const int off = p.foff, nx = p.fnx, ny = p.fny, gx0 = tl.y, gy0 = tl.z;
    const int t = threadIdx.x, lx = t % W1, ly = t / W1, gx = gx0 - 1 + lx, gy = gy0 - 1 + ly;
    const bool in = t < W1 * W1 && gx >= 0 && gx <= nx && gy >= 0 && gy <= ny;
    const int i = in ? off + gx + gy * (nx + 1) : off;
    NodeRow<T> row;
    row.load(i, A, Dinv);
    const bool done = cta_done(fl, tl.x);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    const Vec2<T> bv = lv2(b, i);
    for (int l = t; l < W2 * W2; l += kTileThreads) {
        const int hx = gx0 - 2 + l % W2, hy = gy0 - 2 + l / W2;
        Vec2<T> v;
        v.x = v.y = 0;
        if (hx >= 0 && hx <= nx && hy >= 0 && hy <= ny) {
            const int h = off + hx + hy * (nx + 1);
            v = lv2(x, h);
            const Vec2<T> e = interpolate(hx, hy, p, xc);
            if (!fixed[2 * h]) v.x += e.x;
            if (!fixed[2 * h + 1]) v.y += e.y;
        }
        s2[l] = v;
    }
    __syncthreads();
    const int c = (ly + 1) * W2 + lx + 1;
    if (t < W1 * W1) {
        Vec2<T> v;
        v.x = v.y = 0;
        if (in) v = row.relax(s2[c], row.residual(bv, s2, c, W2));
        s1[t] = v;
    }
    __syncthreads();
    if (in && lx >= 1 && lx <= W0 && ly >= 1 && ly <= W0) {
        const Vec2<T> v = row.relax(s1[t], row.residual(bv, s1, t, W1));
        if (FINE) s0[(ly - 1) * W0 + lx - 1] = v;
        else st2(xo, i, v.x, v.y);
    }
    if (!FINE) return;
    // level 0's x is on its way while the sweep ends
    constexpr int F = 2 * kUpTile, kPer = (F * F + kTileThreads - 1) / kTileThreads;
    Vec2<T> xv[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int l = threadIdx.x + u * kTileThreads, gx = 2 * gx0 + l % F, gy = 2 * gy0 + l / F;
        if (l < F * F && gx <= pf.fnx && gy <= pf.fny) xv[u] = lv2(x0, pf.foff + gx + gy * (pf.fnx + 1));
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int l = threadIdx.x + u * kTileThreads, gx = 2 * gx0 + l % F, gy = 2 * gy0 + l / F;
        if (l >= F * F || gx > pf.fnx || gy > pf.fny) continue;
        int I0, I1, J0, J1;
        parents(gx, pf.fnx, I0, I1);
        parents(gy, pf.fny, J0, J1);
        I0 -= gx0;
        I1 -= gx0;
        J0 -= gy0;
        J1 -= gy0;
        const Vec2<T> a = s0[J0 * W0 + I0], bq = s0[J0 * W0 + I1], c = s0[J1 * W0 + I0], d = s0[J1 * W0 + I1];
        const int i = pf.foff + gx + gy * (pf.fnx + 1);
        Vec2<T> v = xv[u];
        if (!fixed0[2 * i]) v.x += (T)0.25 * ((a.x + bq.x) + (c.x + d.x));
        if (!fixed0[2 * i + 1]) v.y += (T)0.25 * ((a.y + bq.y) + (c.y + d.y));
        st2(x0, i, v.x, v.y);
    }
}

// The levels of at most kBottomNodes nodes of one RVE, down to the coarsest
// and back, in one CTA.  Every thread owns one node of one level (a level
// starts at a warp boundary): its operator row, its place in the transfers
// and its masks are in registers before the wait, and shared memory holds the
// vectors alone.  Bound by the latency of its 16 or so phases, each a block
// barrier and one node's arithmetic.  (With the operators staged in shared
// memory and a loop over each level's nodes the phases took 11 us of 16.)
constexpr int kBottomNodes = 300;
constexpr int kBottomThreads = 512;
constexpr int kBottomLevels = 8;

struct Bottom {
    int nlev, first;                       // levels, and the first one's number in the hierarchy
    int nx[kBottomLevels], ny[kBottomLevels], off[kBottomLevels];
    int thread[kBottomLevels];             // first thread of each level but the coarsest
    int vec[kBottomLevels];                // and its place in the shared vectors
    int foff, fnx, fny;                    // the grid its result is interpolated to when `first` is level 1
};
// Its vectors (right-hand sides, two iterates, the residual of every level):
// at most so many nodes each, with a margin on both sides, as a boundary
// node's row of (zero) blocks reads up to a line of nodes past its level.
constexpr int kBottomVec = 544, kBottomPad = 160, kBottomStride = kBottomVec + 2 * kBottomPad;
static_assert(kBottomVec >= kBottomThreads + (kCoarseCells + 1) * (kCoarseCells + 1), "room for every thread's node");
static_assert(kBottomPad > kBottomNodes / 2 + 1, "a line of the narrowest level");

template <typename T>
struct BottomArrays {                      // of the hierarchy's levels, by number
    const T* A[17];
    const T* Dinv[17];
    const uint8_t* fixed[17];
    const T* b[17];
    T* xo[17];
};

template <typename T>
__global__ void __launch_bounds__(kBottomThreads) k_mg_bottom(const Bottom* __restrict__ bottoms, BottomArrays<T> ar,
                                                              const double* __restrict__ XT,
                                                              const uint8_t* __restrict__ fixed0, T* x0, const int* fl) {
    constexpr int kPad = kBottomPad;
    extern __shared__ __align__(16) unsigned char bottom_smem[];
    Vec2<T>* s_vec = reinterpret_cast<Vec2<T>*>(bottom_smem);
    __shared__ Bottom B;
    __shared__ double s_inv[kCoarseStride];
    __shared__ double s_rhs[kCoarseMaxDof];
    __shared__ double s_part[8][64];
    const int r = blockIdx.x, t = threadIdx.x;
    if (t < (int)(sizeof(Bottom) / sizeof(int)))
        reinterpret_cast<int*>(&B)[t] = reinterpret_cast<const int*>(&bottoms[r])[t];
    for (int q = t; q < 4 * kBottomStride; q += kBottomThreads) {
        Vec2<T> z;
        z.x = z.y = 0;
        s_vec[q] = z;
    }
    __syncthreads();
    const int kc = B.nlev - 1, nc = 2 * (B.nx[kc] + 1) * (B.ny[kc] + 1);
    // the thread's node
    int lev = -1;
    for (int k = 0; k < kc; ++k)
        if (t >= B.thread[k]) lev = k;
    int node = 0, W = 1, nx = 0, ny = 0;
    if (lev >= 0) {
        nx = B.nx[lev];
        ny = B.ny[lev];
        W = nx + 1;
        node = t - B.thread[lev];
        if (node >= W * (ny + 1)) lev = -1;
    }
    NodeRow<T> row;
    int at = kPad, cat = kPad;             // of the node, and of its level's coarser one, in the vectors
    int pa = 0, pb = 0, pc = 0, pd = 0;    // its parents there
    bool f0 = true, f1 = true;             // its masks
    int cn = -1, fat = 0;                  // the coarse node it restricts to: number, and its place on this level
    T wx[3], wy[3];
    bool cf0 = true, cf1 = true;
    if (lev >= 0) {
        const int l = B.first + lev, gx = node % W, gy = node / W;
        row.load(B.off[lev] + node, ar.A[l], ar.Dinv[l]);
        f0 = ar.fixed[l][2 * (size_t)(B.off[lev] + node)];
        f1 = ar.fixed[l][2 * (size_t)(B.off[lev] + node) + 1];
        at = kPad + B.vec[lev] + node;
        cat = kPad + B.vec[lev + 1];
        const int cW = B.nx[lev + 1] + 1, cN = cW * (B.ny[lev + 1] + 1);
        int I0, I1, J0, J1;
        parents(gx, nx, I0, I1);
        parents(gy, ny, J0, J1);
        pa = cat + I0 + J0 * cW;
        pb = cat + I1 + J0 * cW;
        pc = cat + I0 + J1 * cW;
        pd = cat + I1 + J1 * cW;
        if (node < cN) {                   // a level has at least as many nodes as the one below it
            cn = node;
            const int px = grid_pos(cn % cW, nx), py = grid_pos(cn / cW, ny);
            side_weights(px, nx, wx[0], wx[2]);
            side_weights(py, ny, wy[0], wy[2]);
            wx[1] = wy[1] = (T)1;
            fat = kPad + B.vec[lev] + px + py * W;
            cf0 = ar.fixed[l + 1][2 * (size_t)(B.off[lev + 1] + cn)];
            cf1 = ar.fixed[l + 1][2 * (size_t)(B.off[lev + 1] + cn) + 1];
        }
    }
    for (int q = t; q < nc * nc; q += kBottomThreads) s_inv[q] = XT[(size_t)r * kCoarseStride + q];
    Vec2<T>*vb = s_vec, *v1 = vb + kBottomStride, *v2 = v1 + kBottomStride, *vr = v2 + kBottomStride;
    const bool done = cta_done(fl, r);
    pdl_wait();
    pdl_trigger();
    if (done) return;
    {
        const int n = (B.nx[0] + 1) * (B.ny[0] + 1);
        if (t < n) vb[kPad + B.vec[0] + t] = lv2(ar.b[B.first], B.off[0] + t);
    }
    __syncthreads();
    Vec2<T> b, x;
    b.x = b.y = x.x = x.y = 0;
    for (int k = 0; k < kc; ++k) {
        const bool mine = lev == k;
        if (mine) {
            Vec2<T> z;
            z.x = z.y = 0;
            b = vb[at];
            x = row.relax(z, b);
            v1[at] = x;
        }
        __syncthreads();
        if (mine) {
            x = row.relax(x, row.residual(b, v1, at, W));
            v2[at] = x;
        }
        __syncthreads();
        if (mine) vr[at] = row.residual(b, v2, at, W);
        __syncthreads();
        if (mine && cn >= 0) {
            T s0 = 0, s1 = 0;
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx) {
                    const T w = wy[dy + 1] * wx[dx + 1];
                    const Vec2<T> v = vr[fat + dx + dy * W];
                    s0 += w * v.x;
                    s1 += w * v.y;
                }
            Vec2<T> v;
            v.x = cf0 ? (T)0 : s0;
            v.y = cf1 ? (T)0 : s1;
            vb[cat + cn] = v;
        }
        __syncthreads();
    }
    // the coarsest grid: x = X b with the explicit masked inverse, eight threads per DOF
    {
        const T* bc = reinterpret_cast<const T*>(vb + kPad + B.vec[kc]);
        T* xc = reinterpret_cast<T*>(v2 + kPad + B.vec[kc]);
        if (t < nc) s_rhs[t] = (double)bc[t];
        __syncthreads();
        const int q = t % 64, part = t / 64;
        double acc = 0.0;
        if (q < nc)
            for (int j = part; j < nc; j += kBottomThreads / 64) acc += s_inv[j * nc + q] * s_rhs[j];
        s_part[part][q] = acc;
        __syncthreads();
        if (t < nc) {
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < kBottomThreads / 64; ++k) v += s_part[k][t];
            xc[t] = (T)v;
        }
        __syncthreads();
    }
    for (int k = kc - 1; k >= 0; --k) {
        const bool mine = lev == k;
        if (mine) {
            const Vec2<T> a = v2[pa], bq = v2[pb], c = v2[pc], d = v2[pd];
            if (!f0) x.x += (T)0.25 * ((a.x + bq.x) + (c.x + d.x));
            if (!f1) x.y += (T)0.25 * ((a.y + bq.y) + (c.y + d.y));
            vr[at] = x;
        }
        __syncthreads();
        if (mine) {
            x = row.relax(x, row.residual(b, vr, at, W));
            v1[at] = x;
        }
        __syncthreads();
        if (mine) {
            x = row.relax(x, row.residual(b, v1, at, W));
            v2[at] = x;
        }
        __syncthreads();
    }
    const int n0 = (B.nx[0] + 1) * (B.ny[0] + 1);
    const Vec2<T>* xr = v2 + kPad + B.vec[0];
    if (B.first > 1) {
        if (t < n0) st2(ar.xo[B.first], B.off[0] + t, xr[t].x, xr[t].y);
        return;
    }
    const int W0 = B.nx[0] + 1, nf = (B.fnx + 1) * (B.fny + 1);
    for (int l = t; l < nf; l += kBottomThreads) {
        int I0, I1, J0, J1;
        parents(l % (B.fnx + 1), B.fnx, I0, I1);
        parents(l / (B.fnx + 1), B.fny, J0, J1);
        const Vec2<T> a = xr[I0 + J0 * W0], bq = xr[I1 + J0 * W0], c = xr[I0 + J1 * W0], d = xr[I1 + J1 * W0];
        const int i = B.foff + l;
        Vec2<T> v = lv2(x0, i);
        if (!fixed0[2 * i]) v.x += (T)0.25 * ((a.x + bq.x) + (c.x + d.x));
        if (!fixed0[2 * i + 1]) v.y += (T)0.25 * ((a.y + bq.y) + (c.y + d.y));
        st2(x0, i, v.x, v.y);
    }
}

// ---------------------------------------------------------------------------
// Numeric set-up
// ---------------------------------------------------------------------------

// Coarse mask by injection: the coarse node takes the mask of the finer node at its position.
__global__ inline void k_mg_inject_mask(int n, const int* __restrict__ node_rve, const Pair* __restrict__ pair,
                                        const uint8_t* fixed_f, uint8_t* fixed_c) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    const Pair p = pair[node_rve ? node_rve[a] : 0];
    const int la = a - p.coff, I = la % (p.cnx + 1), J = la / (p.cnx + 1);
    const int i = p.foff + grid_pos(I, p.fnx) + grid_pos(J, p.fny) * (p.fnx + 1);
    fixed_c[2 * a] = fixed_f[2 * i];
    fixed_c[2 * a + 1] = fixed_f[2 * i + 1];
}

// inverse of a node's masked diagonal block
__device__ __forceinline__ void masked_inverse(const double b[4], bool f0, bool f1, double m[4]) {
    m[0] = m[1] = m[2] = m[3] = 0.0;
    if (!f0 && !f1) {
        const double det = b[0] * b[3] - b[1] * b[2];
        if (det != 0.0) {
            m[0] = b[3] / det;
            m[1] = -b[1] / det;
            m[2] = -b[2] / det;
            m[3] = b[0] / det;
        }
    } else {
        m[0] = (f0 || b[0] == 0.0) ? 0.0 : 1.0 / b[0];
        m[3] = (f1 || b[3] == 0.0) ? 0.0 : 1.0 / b[3];
    }
}

// Galerkin product A_c = M_c P^T M A M P M_c of one level and its diagonal
// inverses, in FP64, with FP32 copies on request.  A CTA takes 32 coarse
// nodes, a warp one component of one of their nine children each: its lanes'
// rows have the same pattern and the same weights, but at the grid's edge, so
// a block goes only to the one to four coarse blocks it has a weight for.  Sums in registers,
// added through shared memory in the order of the children.  (With the nine
// children of a node in neighbouring lanes every block took the instructions
// of all nine targets: 230 us on level 1 of 512^2 and 152 on the six below;
// now 125 and 82, bound by the instructions of 18 warps per SM.)
constexpr int kGalNodes = 32;
constexpr int kGalThreads = 2 * 9 * kGalNodes;
constexpr int kGalRow = kGalNodes + 1;  // odd: different entries of a node in different banks

template <bool FINE_BSR>
__global__ void __launch_bounds__(kGalThreads) k_mg_galerkin(int n, const int* __restrict__ node_rve,
                                                             const Pair* __restrict__ pair, const int* __restrict__ row_ptr,
                                                             const double* __restrict__ K,
                                                             const double* __restrict__ A,
                                                             const uint8_t* __restrict__ fixed_f,
                                                             const uint8_t* __restrict__ fixed_c, double* __restrict__ Ac,
                                                             float* __restrict__ Acf, double* __restrict__ Dinv,
                                                             float* __restrict__ Dinvf) {
    __shared__ double acc[3][36 * kGalRow];
    const int t = threadIdx.x, a0 = blockIdx.x * kGalNodes, ch = (t >> 5) % 9, d = t / (9 * kGalNodes), node = t & 31;
    double v[9][2];
#pragma unroll
    for (int o = 0; o < 9; ++o) v[o][0] = v[o][1] = 0.0;
    const int a = a0 + node;
    if (a < n) {
        const Pair p = pair[node_rve ? node_rve[a] : 0];
        const int la = a - p.coff, Ia = la % (p.cnx + 1), Ja = la / (p.cnx + 1);
        const int cx = grid_pos(Ia, p.fnx) + ch % 3 - 1, cy = grid_pos(Ja, p.fny) + ch / 3 - 1;
        double wi = 0.0;
        if (cx >= 0 && cx <= p.fnx && cy >= 0 && cy <= p.fny) wi = grid_w(cx, p.fnx, Ia) * grid_w(cy, p.fny, Ja);
        if (wi != 0.0) {
            const int W = p.fnx + 1, i = p.foff + cx + cy * W;
            const double wd = fixed_f[2 * i + d] ? 0.0 : wi;
            // 2 bits per neighbour column (row) and coarse column (row): weight 0, 1 or 1/2 as 0, 1, 2
            auto code = [](int g, int nf, int I) {
                const double w = grid_w(g, nf, I);
                return w == 0.0 ? 0u : w == 1.0 ? 1u : 2u;
            };
            unsigned wx = 0, wy = 0, in = 0;  // in: the neighbours inside the grid
#pragma unroll
            for (int e = 0; e < 9; ++e) {
                wx |= code(cx + e / 3 - 1, p.fnx, Ia + e % 3 - 1) << 2 * e;
                wy |= code(cy + e / 3 - 1, p.fny, Ja + e % 3 - 1) << 2 * e;
                const int gx = cx + e % 3 - 1, gy = cy + e / 3 - 1;
                in |= (gx >= 0 && gx <= p.fnx && gy >= 0 && gy <= p.fny ? 1u : 0u) << e;
            }
            // level 0: the row's first blocks are its grid neighbours in order (no enrichment node has a coarse part)
            const unsigned mask = FINE_BSR ? grid_nbr_mask(cx, cy, p.fnx, p.fny) : in;
            const double* blk = (FINE_BSR ? K + 4 * (size_t)row_ptr[i] : A + 36 * (size_t)i) + 2 * d;
            const uchar2* fix = reinterpret_cast<const uchar2*>(fixed_f) + i;
#pragma unroll
            for (int s = 0; s < 9; s += 3) {
                double b[3][2];
                uchar2 f[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    b[u][0] = b[u][1] = 0.0;
                    if (!(mask >> (s + u) & 1)) continue;
                    const int q = FINE_BSR ? __popc(mask & ((1u << (s + u)) - 1u)) : s + u;
                    load2(blk + 4 * q, b[u][0], b[u][1]);
                    f[u] = fix[(s / 3 - 1) * W + u - 1];
                }
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    if (!(mask >> (s + u) & 1)) continue;
                    const double b0 = f[u].x ? 0.0 : wd * b[u][0], b1 = f[u].y ? 0.0 : wd * b[u][1];
#pragma unroll
                    for (int oy = 0; oy < 3; ++oy) {
                        const unsigned ky = wy >> 2 * (s + oy) & 3u;
                        if (!ky) continue;
#pragma unroll
                        for (int ox = 0; ox < 3; ++ox) {
                            const unsigned kx = wx >> 2 * (3 * u + ox) & 3u;
                            if (!kx) continue;
                            // 2^(2 - kx - ky)
                            const double w = __hiloint2double((int)((1025u - kx - ky) << 20), 0);
                            v[3 * oy + ox][0] += w * b0;
                            v[3 * oy + ox][1] += w * b1;
                        }
                    }
                }
            }
        }
    }
    // a group of three children each, then the groups
#pragma unroll
    for (int turn = 0; turn < 3; ++turn) {
        if (ch % 3 == turn) {
            double* o = acc[ch / 3] + 2 * d * kGalRow + node;
#pragma unroll
            for (int k = 0; k < 9; ++k)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    double& x = o[(4 * k + e) * kGalRow];
                    x = turn ? x + v[k][e] : v[k][e];
                }
        }
        __syncthreads();
    }
    auto total = [&](int k, int nd) { return acc[0][k * kGalRow + nd] + acc[1][k * kGalRow + nd] + acc[2][k * kGalRow + nd]; };
    for (int q = t; q < 36 * kGalNodes; q += kGalThreads) {
        const int nd = q / 36, k = q % 36, c = a0 + nd;
        if (c >= n) break;
        double s = total(k, nd);
        const Pair p = pair[node_rve ? node_rve[c] : 0];
        const int la = c - p.coff, Ib = la % (p.cnx + 1) + k / 4 % 3 - 1, Jb = la / (p.cnx + 1) + k / 12 - 1;
        if (Ib < 0 || Ib > p.cnx || Jb < 0 || Jb > p.cny || fixed_c[2 * c + k % 4 / 2] ||
            fixed_c[2 * (p.coff + Ib + Jb * (p.cnx + 1)) + k % 2])
            s = 0.0;
        Ac[36 * (size_t)c + k] = s;
        if (Acf) Acf[36 * (size_t)c + k] = (float)s;
    }
    if (t < kGalNodes && a0 + t < n) {
        const int c = a0 + t;
        const bool f0 = fixed_c[2 * c], f1 = fixed_c[2 * c + 1];
        double b[4], m[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) b[k] = total(16 + k, t);
        masked_inverse(b, f0, f1, m);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            Dinv[4 * (size_t)c + k] = m[k];
            if (Dinvf) Dinvf[4 * (size_t)c + k] = (float)m[k];
        }
    }
}

__global__ inline void k_mg_to_f32(size_t n, const double* a, float* b) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}

// The coarsest operator of each RVE (one CTA each) inverted explicitly, by
// Gauss-Jordan elimination in place with partial pivoting: fixed DOFs get
// identity rows and columns, and zero rows and columns in the result.  A
// thread keeps its column's rows t / 64, t / 64 + 4, ... in registers; rows
// stay where they are, and step k's pivot is the largest entry of column k in
// a row that no step has taken.  A step's column and pivot row pass through
// shared memory.  Stored transposed (XT[j n + r] = X[r][j]).  Flag 3 = 1 on a
// zero pivot.  Bound by the latency of a step, 50 of them at most.  (With
// [M | I] in shared memory and row exchanges: 102 us, now 64.)
struct Coarse {
    const double* A;
    const uint8_t* fixed;
    int off, nx, ny, pad;
};
constexpr int kFactorThreads = 256;

__global__ void __launch_bounds__(kFactorThreads) k_mg_coarse_inverse(const Coarse* __restrict__ cd, double* XT, int* fl) {
    constexpr int kCols = 64, kRowStep = kFactorThreads / kCols, kPer = (kCoarseMaxDof + kRowStep - 1) / kRowStep;
    static_assert(kCoarseMaxDof <= kCols, "a thread per column");
    constexpr int kW = kCoarseMaxDof + 1;  // odd: a column's entries in different banks
    __shared__ double M[kCoarseMaxDof][kW];
    __shared__ double s_colk[2][kPer * kRowStep], s_row[kCols], s_best[2][kRowStep];
    __shared__ int s_arg[2][kRowStep], s_step[kCoarseMaxDof], s_pivot[kCoarseMaxDof];
    const Coarse C = cd[blockIdx.x];
    const int nn = (C.nx + 1) * (C.ny + 1), n = 2 * nn, t = threadIdx.x;
    const uint8_t* fixed = C.fixed + 2 * (size_t)C.off;
    const double* A = C.A + 36 * (size_t)C.off;
    for (int e = t; e < n * n; e += kFactorThreads) {
        const int r = e / n, c = e % n;
        M[r][c] = c == r && fixed[r] ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int e = t; e < 9 * nn; e += kFactorThreads) {
        const int a = e / 9, o = e % 9, I = a % (C.nx + 1) + o % 3 - 1, J = a / (C.nx + 1) + o / 3 - 1;
        if (I < 0 || I > C.nx || J < 0 || J > C.ny) continue;
        const int b = I + J * (C.nx + 1);
        for (int d = 0; d < 2; ++d)
            for (int f = 0; f < 2; ++f)
                if (!fixed[2 * a + d] && !fixed[2 * b + f]) M[2 * a + d][2 * b + f] = A[36 * (size_t)a + 4 * o + 2 * d + f];
    }
    __syncthreads();
    const int c = t % kCols, rg = t / kCols;
    unsigned taken = 0;  // this thread's rows that were pivots (bit u)
    double v[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int r = rg + u * kRowStep;
        v[u] = r < n && c < n ? M[r][c] : 0.0;
    }
    // column k for the step, and its largest entry among this thread's free rows (the first such row)
    auto publish = [&](int k) {
        if (c != k) return;
        double best = -1.0;
        int arg = n;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int r = rg + u * kRowStep;
            s_colk[k & 1][r] = v[u];
            if (r < n && !(taken >> u & 1)) {
                if (arg == n) arg = r;  // (entries that don't compare: the first free row)
                if (fabs(v[u]) > best) {
                    best = fabs(v[u]);
                    arg = r;
                }
            }
        }
        s_best[k & 1][rg] = best;
        s_arg[k & 1][rg] = arg;
    };
    publish(0);
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        double best = s_best[k & 1][0];
        int pr = s_arg[k & 1][0];
#pragma unroll
        for (int g = 1; g < kRowStep; ++g) {
            const double ob = s_best[k & 1][g];
            const int op = s_arg[k & 1][g];
            if (ob > best || (ob == best && op < pr)) {
                best = ob;
                pr = op;
            }
        }
        const double piv = s_colk[k & 1][pr];
        const int pu = rg == pr % kRowStep ? pr / kRowStep : -1;  // this thread's place of the pivot row
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            if (u == pu) s_row[c] = v[u];
        if (pu >= 0) taken |= 1u << pu;
        if (t == 0) {
            s_step[pr] = k;
            s_pivot[k] = pr;
            if (piv == 0.0) fl[kFlags * blockIdx.x + 3] = 1;
        }
        __syncthreads();
        // column k is replaced by what the unit matrix's column has become
        const double pc = piv != 0.0 ? (c == k ? 1.0 : s_row[c]) / piv : 0.0;
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            v[u] = u == pu ? pc : (c == k ? 0.0 : v[u]) - s_colk[k & 1][rg + u * kRowStep] * pc;
        publish(k + 1);
        __syncthreads();
    }
    // row pr of the result is row s_step[pr] of the inverse, its column k column s_pivot[k]
    double* X = XT + (size_t)blockIdx.x * kCoarseStride;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int r = rg + u * kRowStep;
        if (r >= n || c >= n) continue;
        const int R = s_step[r], J = s_pivot[c];
        X[J * n + R] = (fixed[R] || fixed[J]) ? 0.0 : v[u];
    }
}

// D^-1/2 of a symmetric positive definite block (false if it is not)
__device__ __forceinline__ bool inv_sqrt(const double b[4], double s[4]) {
    const double o = 0.5 * (b[1] + b[2]), det = b[0] * b[3] - o * o, tr = b[0] + b[3];
    if (!(det > 0.0 && tr > 0.0 && isfinite(det))) return false;
    // sqrt(B) = (B + q I) / t, q = sqrt(det), t = sqrt(tr + 2 q); its determinant is q
    const double q = sqrt(det), w = 1.0 / (q * sqrt(tr + 2.0 * q));
    s[0] = (b[3] + q) * w;
    s[1] = s[2] = -o * w;
    s[3] = (b[0] + q) * w;
    return true;
}

// Per RVE the largest block row sum of the scaled enrichment block, max_i
// sum_j ||D_i^-1/2 K_ij D_j^-1/2||_2 >= lambda_max(D^-1 K_ee) (2.2-2.4 on these
// meshes, whose lambda_max is 1.9); infinite when a diagonal block is not
// positive definite.  Kept as the bits of a non-negative double, so the
// maximum does not depend on the order.
__global__ inline void k_enr_bound(int n, const int* __restrict__ node, const int* __restrict__ rve,
                                   const int* __restrict__ reg_end, const int* __restrict__ node_end,
                                   const int* __restrict__ row_ptr, const int* __restrict__ col,
                                   const int* __restrict__ diag, const double* __restrict__ K, unsigned long long* bound) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int i = node[t], r = rve[t], lo = reg_end[r], hi = node_end[r];
    double si[4], sum = 0.0;
    bool ok = inv_sqrt(K + 4 * (size_t)diag[i], si);
    for (int q = row_ptr[i]; ok && q < row_ptr[i + 1]; ++q) {
        const int j = col[q];
        if (j < lo || j >= hi) continue;
        double sj[4];
        ok = inv_sqrt(K + 4 * (size_t)diag[j], sj);
        const double* b = K + 4 * (size_t)q;
        const double u0 = si[0] * b[0] + si[1] * b[2], u1 = si[0] * b[1] + si[1] * b[3];
        const double u2 = si[2] * b[0] + si[3] * b[2], u3 = si[2] * b[1] + si[3] * b[3];
        const double x0 = u0 * sj[0] + u1 * sj[2], x1 = u0 * sj[1] + u1 * sj[3];
        const double x2 = u2 * sj[0] + u3 * sj[2], x3 = u2 * sj[1] + u3 * sj[3];
        const double f = x0 * x0 + x1 * x1 + x2 * x2 + x3 * x3, d = x0 * x3 - x1 * x2;
        sum += sqrt(0.5 * (f + sqrt(fmax(f * f - 4.0 * d * d, 0.0))));
    }
    if (!ok || !isfinite(sum)) sum = INFINITY;
    atomicMax(&bound[r], (unsigned long long)__double_as_longlong(sum));
}

// The Chebyshev recurrence's factors (Saad, Iterative Methods for Sparse
// Linear Systems, Alg. 12.1) for the spectrum (b / kChebRatio, b), b the bound
// with a margin; one damped Jacobi sweep (1/2) where there is no bound.
__global__ inline void k_enr_coef(int nr, const unsigned long long* bound, double* coef) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nr) return;
    const double b = 1.01 * __longlong_as_double((long long)bound[r]);
    double* c = coef + kChebCoef * r;
    if (!(b > 0.0) || !isfinite(b)) {
        c[0] = 0.5;
        for (int k = 1; k < kChebCoef; ++k) c[k] = 0.0;
        return;
    }
    const double theta = 0.5 * (b + b / kChebRatio), delta = 0.5 * (b - b / kChebRatio), sigma = theta / delta;
    double rho = 1.0 / sigma;
    c[0] = 1.0 / theta;
    for (int k = 1; k < kChebSteps; ++k) {
        const double rho1 = 1.0 / (2.0 * sigma - rho);
        c[2 * k - 1] = rho1 * rho;
        c[2 * k] = 2.0 * rho1 / delta;
        rho = rho1;
    }
}

}  // namespace mg
}  // namespace pgb
