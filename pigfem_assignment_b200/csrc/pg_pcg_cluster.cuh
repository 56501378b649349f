// Preconditioned CG of a small system in one launch (see k_pcg_cluster).
#pragma once

#include "pg_solve_kernels.cuh"

namespace pgb {

// All iterations of CG on a system that one cluster of 16 CTAs holds: the
// rows are cut into 16 runs of about as many blocks of K; a CTA keeps its
// rows' vectors, columns and (KS) blocks in shared memory.  For the columns
// of other CTAs' rows (its halo) it fetches z once an iteration through
// distributed shared memory and carries their p = z + beta p along, so the
// matrix product reads local shared memory only.  An iteration has two
// cluster barriers, each of which also carries a dot product: every CTA
// writes its partial into all 16, and each adds them in rank order, so all
// take the same decisions and the result is the same bits on every run.
//
// Three launches per iteration with fused sums take 17.2 us at 64^2 (4.5k
// nodes), nearly all of it launch, fence and ticket latency; with z and p
// gathered remotely for every entry (131 KB a CTA) this kernel took 6.0; as it
// is, 4.2 (3.6 were the two barriers and sums), and 9.1 at 128^2 (17k nodes, K
// from L2) against 17.8.
constexpr int kClusterCtas = 16;
constexpr int kClusterThreads = 384;     // one row each at 64^2 (281 a CTA); 1,024 threads: 5.8 us an iteration, 384: 4.3
constexpr int kClusterUnroll = 4;        // blocks a row loads at once
constexpr unsigned kRowMask = 0x3fffffffu;  // row starts carry the row's two masks above it

struct ClusterCgArgs {
    int n;
    const int* row_ptr;
    const int* col;
    const uint8_t* fixed;
    const double* r;                     // residual at x
    double* x;
    const double* minv;
    double tol2;
    int max_iter;
    int* flags;                          // F_DONE, F_BREAKDOWN, F_ITERS
    double* scal;                        // r.r at the end
    int rows, blocks, halo;              // what a CTA has room for
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_addr(unsigned a, unsigned rank) {
    unsigned o;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(rank));
    return o;
}
__device__ __forceinline__ double2 peer_ld2(unsigned a) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void peer_st(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// one block of K in shared memory, in 128-bit loads
__device__ __forceinline__ void smem_block(const double* p, double& a, double& b, double& c, double& d) {
    const double2 u = reinterpret_cast<const double2*>(p)[0], v = reinterpret_cast<const double2*>(p)[1];
    a = u.x;
    b = u.y;
    c = v.x;
    d = v.y;
}
__device__ __forceinline__ void smem_block(const float* p, double& a, double& b, double& c, double& d) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = v.x;
    b = v.y;
    c = v.z;
    d = v.w;
}

// first row of CTA k: the first whose blocks start at or after k / 16 of all blocks
__host__ __device__ inline int cluster_first_row(const int* row_ptr, int n, int k) {
    if (k <= 0) return 0;
    if (k >= kClusterCtas) return n;
    const long long want = (long long)row_ptr[n] * k / kClusterCtas;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (row_ptr[mid] < want) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Shared memory of k_pcg_cluster: z, r, x, q, p (with the halo's), M^-1, blocks (k_bytes each value; 0: not kept),
// the halo's addresses, row starts, columns (16 bits).  While it sets up, the vectors' place holds a 16-bit map over
// all rows (32 bytes per row of the largest CTA would do; the vectors take 80).
inline size_t cluster_cg_smem(int rows, int blocks, int halo, size_t k_bytes) {
    return (size_t)rows * (5 * 16 + 32) + (size_t)halo * 16 + (size_t)blocks * 4 * k_bytes + (size_t)halo * 4 +
           (size_t)rows * 4 + 16 + (size_t)blocks * 2;
}

template <typename MT, bool KS>
__global__ void __launch_bounds__(kClusterThreads, 1) k_pcg_cluster(ClusterCgArgs a, const MT* __restrict__ K) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    __shared__ int s_lo[kClusterCtas + 1];
    __shared__ int s_scan[kClusterThreads / 32];
    __shared__ double s_red[2][kClusterThreads / 32];
    __shared__ double s_part[3][kClusterCtas];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned me = cluster_rank();
    double2* z = reinterpret_cast<double2*>(cl_smem);
    double2* r = z + a.rows;
    double2* x = r + a.rows;
    double2* q = x + a.rows;
    double2* p = q + a.rows;             // own rows, then the halo
    double4* M = reinterpret_cast<double4*>(p + a.rows + a.halo);
    MT* sK = reinterpret_cast<MT*>(M + a.rows);
    unsigned* shalo = reinterpret_cast<unsigned*>(sK + (KS ? 4 * (size_t)a.blocks : 0));
    unsigned* srow = shalo + a.halo;
    unsigned short* scol = reinterpret_cast<unsigned short*>(srow + a.rows + 4);
    unsigned short* map = reinterpret_cast<unsigned short*>(cl_smem);
    if (t <= kClusterCtas) s_lo[t] = cluster_first_row(a.row_ptr, a.n, t);
    __syncthreads();
    const int lo = s_lo[me], rows = s_lo[me + 1] - lo;
    const int b0 = a.row_ptr[lo], nb = a.row_ptr[lo + rows] - b0;
    for (int k = t; k <= rows; k += kClusterThreads) {
        unsigned v = (unsigned)(a.row_ptr[lo + k] - b0);
        if (k < rows) v |= (a.fixed[2 * (lo + k)] ? 1u << 30 : 0u) | (a.fixed[2 * (lo + k) + 1] ? 1u << 31 : 0u);
        srow[k] = v;
    }
    // the halo: the distinct columns of other CTAs, in ascending order
    for (int k = t; k < a.n; k += kClusterThreads) map[k] = 0;
    __syncthreads();
    for (int k = t; k < nb; k += kClusterThreads) {
        const int c = a.col[b0 + k];
        if (c < lo || c >= lo + rows) map[c] = 1;
    }
    __syncthreads();
    const int chunk = (a.n + kClusterThreads - 1) / kClusterThreads, c0 = min(a.n, t * chunk), c1 = min(a.n, c0 + chunk);
    int cnt = 0;
    for (int c = c0; c < c1; ++c) cnt += map[c];
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    int at = incl - cnt, halo = 0;
    for (int w = 0; w < kClusterThreads / 32; ++w) {
        if (w < warp) at += s_scan[w];
        halo += s_scan[w];
    }
    const unsigned za = smem_addr(z);
    for (int c = c0; c < c1; ++c) {
        if (!map[c]) continue;
        int rk = 0;
#pragma unroll
        for (int s = kClusterCtas / 2; s > 0; s >>= 1)
            if (c >= s_lo[rk + s]) rk += s;
        shalo[at] = peer_addr(za + 16u * (unsigned)(c - s_lo[rk]), (unsigned)rk);
        map[c] = (unsigned short)(a.rows + at);
        ++at;
    }
    __syncthreads();
    for (int k = t; k < nb; k += kClusterThreads) {
        const int c = a.col[b0 + k];
        scol[k] = c < lo || c >= lo + rows ? map[c] : (unsigned short)(c - lo);
    }
    if (KS)
        for (int k = t; k < 4 * nb; k += kClusterThreads) sK[k] = K[4 * (size_t)b0 + k];
    __syncthreads();  // the map is done with
    // both sums of one reduction to every CTA, and the cluster barrier
    auto share = [&](double u, double v, int slot, bool two) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            u += __shfl_down_sync(0xffffffffu, u, o);
            if (two) v += __shfl_down_sync(0xffffffffu, v, o);
        }
        if (lane == 0) {
            s_red[0][warp] = u;
            if (two) s_red[1][warp] = v;
        }
        __syncthreads();
        if (warp == 0) {
            u = lane < kClusterThreads / 32 ? s_red[0][lane] : 0.0;
            v = two && lane < kClusterThreads / 32 ? s_red[1][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                u += __shfl_xor_sync(0xffffffffu, u, o);
                if (two) v += __shfl_xor_sync(0xffffffffu, v, o);
            }
            if (lane < kClusterCtas) {
                peer_st(peer_addr(smem_addr(&s_part[slot][me]), lane), u);
                if (two) peer_st(peer_addr(smem_addr(&s_part[slot + 1][me]), lane), v);
            }
        }
        cluster_barrier();
    };
    auto total = [&](int slot) {
        double v = s_part[slot][lane % kClusterCtas];
#pragma unroll
        for (int o = kClusterCtas / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    double prz = 0.0, prr = 0.0;
    for (int l = t; l < rows; l += kClusterThreads) {
        const int i = lo + l;
        const double r0 = a.r[2 * i], r1 = a.r[2 * i + 1];
        const double* m = a.minv + 4 * (size_t)i;
        const double4 mv = make_double4(m[0], m[1], m[2], m[3]);
        const double2 zv = make_double2(mv.x * r0 + mv.y * r1, mv.z * r0 + mv.w * r1);
        r[l] = make_double2(r0, r1);
        x[l] = make_double2(a.x[2 * i], a.x[2 * i + 1]);
        M[l] = mv;
        z[l] = zv;
        p[l] = make_double2(0.0, 0.0);
        prz += r0 * zv.x + r1 * zv.y;
        prr += r0 * r0 + r1 * r1;
    }
    for (int l = t; l < halo; l += kClusterThreads) p[a.rows + l] = make_double2(0.0, 0.0);
    cluster_barrier();  // every CTA has started: its shared memory may be written
    share(prz, prr, 1, true);
    double rz = total(1), rr = total(2), beta = 0.0;
    int it = 0;
    bool done = rr <= a.tol2, breakdown = false;
    while (!done && it < a.max_iter) {
        for (int l = t; l < halo + rows; l += kClusterThreads) {
            // the halo first: its loads travel while the own rows are computed
            const bool own = l >= halo;
            const int j = own ? l - halo : a.rows + l;
            const double2 zv = own ? z[j] : peer_ld2(shalo[l]);
            double2 pv = p[j];
            pv.x = zv.x + beta * pv.x;
            pv.y = zv.y + beta * pv.y;
            p[j] = pv;
        }
        __syncthreads();
        double acc = 0.0;
        for (int l = t; l < rows; l += kClusterThreads) {
            const unsigned r0 = srow[l];
            const int k1 = (int)(srow[l + 1] & kRowMask);
            double y0 = 0.0, y1 = 0.0;
            for (int kb = (int)(r0 & kRowMask); kb < k1; kb += kClusterUnroll) {
                double kv[kClusterUnroll][4];
                double2 pj[kClusterUnroll];
#pragma unroll
                for (int u = 0; u < kClusterUnroll; ++u) {
                    const int k = kb + u;
                    kv[u][0] = kv[u][1] = kv[u][2] = kv[u][3] = 0.0;
                    pj[u] = make_double2(0.0, 0.0);
                    if (k < k1) {
                        if (KS) smem_block(sK + 4 * (size_t)k, kv[u][0], kv[u][1], kv[u][2], kv[u][3]);
                        else load_block(K + 4 * (size_t)(b0 + k), kv[u][0], kv[u][1], kv[u][2], kv[u][3]);
                        pj[u] = p[scol[k]];
                    }
                }
#pragma unroll
                for (int u = 0; u < kClusterUnroll; ++u) {
                    y0 += kv[u][0] * pj[u].x + kv[u][1] * pj[u].y;
                    y1 += kv[u][2] * pj[u].x + kv[u][3] * pj[u].y;
                }
            }
            if (r0 >> 30 & 1u) y0 = 0.0;
            if (r0 >> 31) y1 = 0.0;
            q[l] = make_double2(y0, y1);
            acc += p[l].x * y0 + p[l].y * y1;
        }
        share(acc, 0.0, 0, false);
        const double pq = total(0);
        if (!(pq > 0.0)) {
            breakdown = true;
            break;
        }
        const double alpha = rz / pq;
        prz = prr = 0.0;
        for (int l = t; l < rows; l += kClusterThreads) {
            const double2 pv = p[l], qv = q[l];
            double2 xv = x[l], rv = r[l];
            const double4 mv = M[l];
            xv.x += alpha * pv.x;
            xv.y += alpha * pv.y;
            rv.x -= alpha * qv.x;
            rv.y -= alpha * qv.y;
            const double2 zv = make_double2(mv.x * rv.x + mv.y * rv.y, mv.z * rv.x + mv.w * rv.y);
            x[l] = xv;
            r[l] = rv;
            z[l] = zv;
            prz += rv.x * zv.x + rv.y * zv.y;
            prr += rv.x * rv.x + rv.y * rv.y;
        }
        share(prz, prr, 1, true);
        const double rzn = total(1);
        rr = total(2);
        beta = rzn / rz;
        rz = rzn;
        ++it;
        done = rr <= a.tol2;
    }
    for (int l = t; l < rows; l += kClusterThreads) {
        const double2 xv = x[l];
        a.x[2 * (lo + l)] = xv.x;
        a.x[2 * (lo + l) + 1] = xv.y;
    }
    if (me == 0 && t == 0) {
        a.flags[F_DONE] = done ? 1 : 0;
        a.flags[F_BREAKDOWN] = breakdown ? 1 : 0;
        a.flags[F_ITERS] = it;
        a.scal[S_AUX] = rr;
    }
    cluster_barrier();  // no CTA leaves while another may read its shared memory
}

}  // namespace pgb
