// Per-node MLP of the learned Newton warm start: BF16 tensor-core (tcgen05)
// forward, backward and weight-gradient kernels with FP32 accumulation in
// tensor memory, plus an FP32 Adam step.  The reference has no learned
// component; the network is a 16 -> 64 -> 64 -> 16 ReLU MLP (two outputs used)
// over per-node features of a load step.
//
// One CTA (4 warps, 128 threads) owns a 128-row tile of nodes: thread t holds
// row t.  Every GEMM is D[128 x N] (+)= A[128 x K] * B[N x K]^T issued by one
// thread as tcgen05.mma.cta_group::1.kind::f16 (BF16 x BF16 -> FP32) with both
// operands in shared memory in the canonical K-major layout without swizzle:
// 8-row x 16-byte core matrices, K-adjacent core matrices 128 B apart (LBO),
// 8-row groups SBO = (K/8)*128 B apart.  D lives in tensor memory (lane = row,
// one 32-bit column per output) and is read back with tcgen05.ld 32x32b.
// Completion is signalled by tcgen05.commit to an mbarrier whose wait is
// bounded; on timeout the kernel records an error, frees its tensor memory
// and returns.
//
// A tile is a chain of GEMMs that wait for one another, so what counts is how
// many tiles an SM has in flight.  Inference (k_mlp_forward) therefore has a
// kernel of its own with one 16 KB operand buffer and 64 columns of tensor
// memory per CTA, seven CTAs per SM: 2^20 rows in 56 us (the L1 and shared
// memory 70% busy, the tensor pipe 11%, DRAM 15%), where the training kernel's
// shape (182 KB, 512 columns, one CTA per SM) took 181.  The BF16
// operand images of the weights are kept beside the FP32 masters (k_pack and
// the optimizer step write them), so a CTA copies them instead of converting.
//
// Weight gradients: dW2 and dW1 come out of one M=128 GEMM whose A stacks
// dZ2^T over dZ1^T and whose B stacks H1^T over X^T (the off-diagonal blocks
// are not read); dW3 uses A = [dY^T; 0].  They accumulate in tensor memory
// over all tiles a CTA processes; each CTA then writes its part of the
// gradient to its own slot and k_grad_sum adds the parts in CTA order.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "pg_internal.cuh"
#include "pg_pdl.cuh"

namespace pgb {
namespace mlp {

constexpr int IN = 16, HID = 64, OUT = 16, USED = 2, TILE = 128, NT = 128;
constexpr uint32_t TMEM_COLS = 512;
// tensor-memory columns
constexpr uint32_t C_Z1 = 0, C_Z2 = 64, C_DW12 = 256, C_DW3 = 384, C_Y = 128;

// BF16 operand images of the weights (bytes from the image's start): W1, W2,
// W3, then the transposes the backward pass multiplies by
constexpr uint32_t P_W1 = 0;                      // B  64 x 16        2 KB
constexpr uint32_t P_W2 = P_W1 + 2048;            // B  64 x 64        8 KB
constexpr uint32_t P_W3 = P_W2 + 8192;            // B  16 x 64        2 KB
constexpr uint32_t P_FORWARD = P_W3 + 2048;       // what inference needs
constexpr uint32_t P_W3T = P_FORWARD;             // B  64 x 16        2 KB
constexpr uint32_t P_W2T = P_W3T + 2048;          // B  64 x 64        8 KB
constexpr uint32_t P_BYTES = P_W2T + 8192;

// shared-memory map of the training kernel (bytes from the 1024-aligned dynamic base)
constexpr uint32_t O_W = 0;                       // the image
constexpr uint32_t O_W1 = O_W + P_W1, O_W2 = O_W + P_W2, O_W3 = O_W + P_W3, O_W3T = O_W + P_W3T, O_W2T = O_W + P_W2T;
constexpr uint32_t O_X = O_W + 22528;             // A 128 x 16        4 KB
constexpr uint32_t O_H1 = O_X + 4096;             // A 128 x 64       16 KB
constexpr uint32_t O_H2 = O_H1 + 16384;           // A 128 x 64       16 KB
constexpr uint32_t O_DY = O_H2 + 16384;           // A 128 x 16        4 KB
constexpr uint32_t O_DZ2 = O_DY + 4096;           // A 128 x 64       16 KB
constexpr uint32_t O_AT = O_DZ2 + 16384;          // A 128 x 128 (dZ2^T ; dZ1^T)   32 KB
constexpr uint32_t O_BT = O_AT + 32768;           // B  80 x 128 (H1^T ; X^T)      20 KB
constexpr uint32_t O_A3 = O_BT + 20480;           // A 128 x 128 (dY^T ; 0)        32 KB
constexpr uint32_t O_B3 = O_A3 + 32768;           // B  64 x 128 (H2^T)            16 KB
static_assert(P_BYTES <= O_X - O_W, "the image's place");
// The allocation also covers O_B3 + 32 KB: every operand's core-matrix grid
// (rows/8 x K/8 groups of 128 B) read with either stride interpretation stays
// inside the allocation.
constexpr uint32_t SMEM_ALLOC = O_B3 + 32768 + 1024;
// and of the inference kernel: the image, one A operand (X, H1 and H2 in turn), the biases
constexpr uint32_t F_W = 0, F_A = F_W + P_FORWARD, F_B = F_A + 16384;
constexpr uint32_t F_ALLOC = F_B + 4 * (HID + HID + OUT) + 1024;
constexpr uint32_t F_COLS = 64;
constexpr int kForwardCtasPerSm = 7;

struct Params {
    float* W1; float* b1; float* W2; float* b2; float* W3; float* b3;
};

constexpr int kW1 = HID * IN, kB1 = HID, kW2 = HID * HID, kB2 = HID, kW3 = OUT * HID, kB3 = OUT;
constexpr int kNParams = kW1 + kB1 + kW2 + kB2 + kW3 + kB3;
constexpr int kParamBlocks = (kNParams + 255) / 256;  // of 256 threads, one per parameter

__host__ __device__ inline Params carve(float* base) {
    Params q;
    q.W1 = base;
    q.b1 = q.W1 + kW1;
    q.W2 = q.b1 + kB1;
    q.b2 = q.W2 + kW2;
    q.W3 = q.b2 + kB2;
    q.b3 = q.W3 + kW3;
    return q;
}

// Sum over a warp's lanes by a fixed butterfly: every lane gets the same
// value, in the same order on every run.
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// byte offset of element (row, k) in a canonical K-major tile with K columns
__device__ __forceinline__ uint32_t kmaj(int row, int k, int K) {
    return (uint32_t)((row >> 3) * (K * 16) + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, int K) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((128u >> 4) & 0x3FFFu) << 16;                 // LBO: K-adjacent core matrices
    d |= (uint64_t)(((uint32_t)(K * 16) >> 4) & 0x3FFFu) << 32;   // SBO: 8-row groups
    d |= (uint64_t)1 << 46;                                       // descriptor version (sm_100)
    return d;                                                     // base offset 0, no swizzle
}

__device__ __forceinline__ uint32_t idesc_bf16(int M, int N) {
    return (1u << 4)                       // D: FP32
           | (1u << 7)                     // A: BF16
           | (1u << 10)                    // B: BF16
           | ((uint32_t)(N >> 3) << 17)    // N
           | ((uint32_t)(M >> 4) << 24);   // M (A, B K-major; no negation)
}

__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

constexpr int kPollLimit = 1 << 22;  // polls of a completion wait before it gives up

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase, int polls) {
    for (int it = 0; it < polls; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void st_bf16(uint8_t* base, uint32_t off, float v) {
    *reinterpret_cast<__nv_bfloat16*>(base + off) = __float2bfloat16_rn(v);
}

// thread's row of a K-major A tile: K/8 16-byte stores
__device__ __forceinline__ void st_row(uint8_t* base, int row, const float* v, int K) {
    for (int c = 0; c < K / 8; ++c) {
        __align__(16) __nv_bfloat16 h[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = __float2bfloat16_rn(v[8 * c + i]);
        *reinterpret_cast<uint4*>(base + kmaj(row, 8 * c, K)) = *reinterpret_cast<const uint4*>(h);
    }
}

// parameter i as BF16 into its places in the operand images
__device__ __forceinline__ void pack_param(uint8_t* img, int i, float v) {
    if (i < kW1) {
        st_bf16(img, P_W1 + kmaj(i / IN, i % IN, IN), v);
        return;
    }
    i -= kW1 + kB1;
    if (i >= 0 && i < kW2) {
        st_bf16(img, P_W2 + kmaj(i / HID, i % HID, HID), v);
        st_bf16(img, P_W2T + kmaj(i % HID, i / HID, HID), v);
    }
    i -= kW2 + kB2;
    if (i >= 0 && i < kW3) {
        st_bf16(img, P_W3 + kmaj(i / HID, i % HID, HID), v);
        st_bf16(img, P_W3T + kmaj(i % HID, i / HID, OUT), v);
    }
}

__global__ void k_pack(const float* p, uint8_t* img) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNParams) pack_param(img, i, p[i]);
}

// How the completion waits of one launch behave: polls before a wait gives
// up, and (self-test only) a GEMM whose MMAs are not issued, so that nothing
// ever arrives on its mbarrier and its wait must run out.
struct WaitCfg {
    int polls;
    int skip_gemm;  // index of the GEMM not issued, -1: none
};

// Issues the K/16 MMAs of one GEMM (thread 0) and waits for them (all threads).
// Returns false on a timed-out wait; `inflight` then says whether MMAs of this
// CTA are still pending on the phase `phase` (left unflipped).
__device__ __forceinline__ bool gemm(uint32_t sbase, uint32_t a_off, uint32_t b_off, int K, int N, uint32_t d_tmem,
                                     bool accumulate, uint32_t mbar, uint32_t& phase, const WaitCfg& wc, int& index,
                                     bool& inflight) {
    const bool issue = index++ != wc.skip_gemm;
    fence_async_smem();
    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && issue) {
        fence_after();
        const uint32_t id = idesc_bf16(128, N);
        for (int ks = 0; ks < K / 16; ++ks) {
            const uint64_t a = sdesc(sbase + a_off + 256u * ks, K);
            const uint64_t b = sdesc(sbase + b_off + 256u * ks, K);
            umma(d_tmem, a, b, id, (accumulate || ks > 0) ? 1u : 0u);
        }
        umma_commit(mbar);
    }
    bool ok = mbar_wait(mbar, phase, wc.polls);
    ok = __syncthreads_and(ok) != 0;  // every thread takes the same branch afterwards
    if (!ok) {
        inflight = issue;
        return false;
    }
    phase ^= 1u;
    fence_after();
    return ok;
}

__device__ __forceinline__ void mbar_init(uint32_t mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
template <uint32_t COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(slot)),
                 "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <uint32_t COLS>
__device__ __forceinline__ void tmem_free(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
}

__device__ __forceinline__ void tmem_ld2(uint32_t taddr, float* v) {
    uint32_t r0, r1;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    v[0] = __uint_as_float(r0);
    v[1] = __uint_as_float(r1);
}

// 32 consecutive columns of the thread's row
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
#define PG_R(i) "=r"(r[i])
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : PG_R(0), PG_R(1), PG_R(2), PG_R(3), PG_R(4), PG_R(5), PG_R(6), PG_R(7), PG_R(8), PG_R(9), PG_R(10), PG_R(11),
          PG_R(12), PG_R(13), PG_R(14), PG_R(15), PG_R(16), PG_R(17), PG_R(18), PG_R(19), PG_R(20), PG_R(21), PG_R(22),
          PG_R(23), PG_R(24), PG_R(25), PG_R(26), PG_R(27), PG_R(28), PG_R(29), PG_R(30), PG_R(31)
        : "r"(taddr));
#undef PG_R
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Row r of a tile (unsigned: inference asks for the rows of one tile past the
// last, up to 255 beyond the largest number of rows)
__host__ __device__ constexpr unsigned tile_row(int tile, int r) { return (unsigned)tile * TILE + r; }
static_assert(tile_row(INT_MAX / TILE + 1, TILE - 1) > INT_MAX, "no row past the end wraps to one before it");

// The thread's share of a tile of X, 16 floats.  VEC (X is 16-byte aligned):
// four 16-byte loads, each of a warp's 32 covering 512 consecutive bytes, so
// its share is a quarter of the rows 32 warp + 8 k + lane / 4; otherwise its
// own row.
template <bool VEC>
__device__ __forceinline__ void load_x(const float* __restrict__ X, int tile, int n, float* x) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (VEC) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned row = tile_row(tile, 32 * warp + 8 * k + lane / 4);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < (unsigned)n) v = __ldg(reinterpret_cast<const float4*>(X + (size_t)row * IN) + lane % 4);
            x[4 * k] = v.x;
            x[4 * k + 1] = v.y;
            x[4 * k + 2] = v.z;
            x[4 * k + 3] = v.w;
        }
    } else {
        const unsigned row = tile_row(tile, tid);
#pragma unroll
        for (int i = 0; i < IN; ++i) x[i] = row < (unsigned)n ? X[(size_t)row * IN + i] : 0.f;
    }
}
// and into the A operand
template <bool VEC>
__device__ __forceinline__ void store_x(uint8_t* base, const float* x) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (VEC) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            __align__(8) __nv_bfloat162 h[2];
            h[0] = __floats2bfloat162_rn(x[4 * k], x[4 * k + 1]);
            h[1] = __floats2bfloat162_rn(x[4 * k + 2], x[4 * k + 3]);
            *reinterpret_cast<uint2*>(base + kmaj(32 * warp + 8 * k + lane / 4, 4 * (lane % 4), IN)) =
                *reinterpret_cast<const uint2*>(h);
        }
    } else {
        st_row(base, tid, x, IN);
    }
}

// Inference over n rows.  The next tile's row is loaded while this one's
// GEMMs run; a layer is read back 32 columns at a time and stored at once as
// the next layer's operand, over the one the finished GEMM has read.
template <bool VEC>
__global__ void __launch_bounds__(NT, kForwardCtasPerSm) k_mlp_forward(const float* __restrict__ X, int n, Params p,
                                                                       const uint4* __restrict__ img, float* Y_out, int* err,
                                                                       WaitCfg wc) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    __shared__ __align__(8) uint64_t mbar_storage;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&mbar_storage);
    float* sb = reinterpret_cast<float*>(sm + F_B);  // b1, b2, b3
    const int ntiles = (n + TILE - 1) / TILE;
    float x[IN];
    load_x<VEC>(X, blockIdx.x, n, x);
    for (uint32_t i = tid; i < P_FORWARD / 16; i += NT) reinterpret_cast<uint4*>(sm + F_W)[i] = img[i];
    if (tid < HID) {
        sb[tid] = p.b1[tid];
        sb[HID + tid] = p.b2[tid];
    }
    if (tid < OUT) sb[2 * HID + tid] = p.b3[tid];
    if (tid == 0) mbar_init(mbar);
    if (warp == 0) tmem_alloc<F_COLS>(&tmem_slot);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    uint32_t phase = 0;
    bool ok = true;
    int gi = 0;             // GEMMs issued so far (WaitCfg::skip_gemm)
    bool inflight = false;  // a timed-out wait left MMAs of this CTA pending
    // relu(accumulator + bias) of the thread's row as the next operand
    auto hidden = [&](const float* bias) {
#pragma unroll
        for (int c = 0; c < HID; c += 32) {
            float z[32];
            tmem_ld32(tmem + lane_base + c, z);
#pragma unroll
            for (int q = 0; q < 32; q += 8) {
                __align__(16) __nv_bfloat162 h[4];
                const float4 b0 = *reinterpret_cast<const float4*>(bias + c + q);
                const float4 b1 = *reinterpret_cast<const float4*>(bias + c + q + 4);
                h[0] = __floats2bfloat162_rn(fmaxf(z[q] + b0.x, 0.f), fmaxf(z[q + 1] + b0.y, 0.f));
                h[1] = __floats2bfloat162_rn(fmaxf(z[q + 2] + b0.z, 0.f), fmaxf(z[q + 3] + b0.w, 0.f));
                h[2] = __floats2bfloat162_rn(fmaxf(z[q + 4] + b1.x, 0.f), fmaxf(z[q + 5] + b1.y, 0.f));
                h[3] = __floats2bfloat162_rn(fmaxf(z[q + 6] + b1.z, 0.f), fmaxf(z[q + 7] + b1.w, 0.f));
                *reinterpret_cast<uint4*>(sm + F_A + kmaj(tid, c + q, HID)) = *reinterpret_cast<const uint4*>(h);
            }
        }
    };
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int row = tile * TILE + tid;
        store_x<VEC>(sm + F_A, x);
        load_x<VEC>(X, min(tile + (int)gridDim.x, ntiles), n, x);  // (past the last tile: nothing)
        ok = gemm(sbase, F_A, F_W + P_W1, IN, HID, tmem, false, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        hidden(sb);
        ok = gemm(sbase, F_A, F_W + P_W2, HID, HID, tmem, false, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        hidden(sb + HID);
        ok = gemm(sbase, F_A, F_W + P_W3, HID, OUT, tmem, false, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        float y[2];
        tmem_ld2(tmem + lane_base, y);
        if (row < n) {
            const float y0 = y[0] + sb[2 * HID], y1 = y[1] + sb[2 * HID + 1];
            if (VEC) {
                *reinterpret_cast<float2*>(Y_out + 2 * (size_t)row) = make_float2(y0, y1);
            } else {
                Y_out[2 * (size_t)row] = y0;
                Y_out[2 * (size_t)row + 1] = y1;
            }
        }
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    // MMAs still pending after a timed-out wait write tensor memory: wait for
    // them (bounded again) before that memory is freed below
    if (!ok && inflight) mbar_wait(mbar, phase, kPollLimit);
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_free<F_COLS>(tmem);
}

// Sums of 32 values over a warp's lanes, all at once: lane l ends with the
// sum of v[l], by the pairing of a butterfly (the lanes 16 apart first).  31
// exchanges, where a butterfly per value takes 160.
__device__ __forceinline__ float warp_sum32(float* v, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool hi = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float send = hi ? v[i] : v[i + o], keep = hi ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

// Training pass over n rows: this CTA's gradient (kNParams floats, summed
// over its tiles) to gpart + CTA * kNParams and its share of the loss to
// lpart[CTA]; the CTAs' parts are added in CTA order by the next kernel.
// Every sum inside a CTA has a fixed order too (warp butterflies, then the
// four warps in order, then the tiles in order), so a gradient is the same
// bits on every run.
__global__ void __launch_bounds__(NT, 1) k_mlp_train(const float* __restrict__ X, const float* __restrict__ T, int n,
                                                     Params p, const uint4* img, float* gpart, double* lpart,
                                                     int* err, WaitCfg wc) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    __shared__ __align__(8) uint64_t mbar_storage;
    __shared__ uint32_t tmem_slot;
    constexpr int NB = HID + HID + OUT;  // bias gradients: b1, b2, b3
    __shared__ float sgb[NB];
    __shared__ float sbias[NB];
    __shared__ float sloss;
    __shared__ float swarp[NT / 32][NB + 1];  // per warp: this tile's bias-gradient and loss sums
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&mbar_storage);

    for (int i = tid; i < 32768 / 16; i += NT) reinterpret_cast<uint4*>(sm + O_A3)[i] = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < NB; i += NT) sgb[i] = 0.f;
    for (int i = tid; i < (NT / 32) * (NB + 1); i += NT) (&swarp[0][0])[i] = 0.f;
    if (tid == 0) sloss = 0.f;
    if (tid == 0) mbar_init(mbar);
    if (warp == 0) tmem_alloc<TMEM_COLS>(&tmem_slot);
    // the minibatch before has stepped the network (and read the parts that this one writes)
    pdl_wait();
    pdl_trigger();
    const int failed = __ldcg(err);
    for (uint32_t i = tid; i < P_BYTES / 16; i += NT) reinterpret_cast<uint4*>(sm + O_W)[i] = __ldcg(&img[i]);
    if (tid < HID) {
        sbias[tid] = __ldcg(&p.b1[tid]);
        sbias[HID + tid] = __ldcg(&p.b2[tid]);
    }
    if (tid < OUT) sbias[2 * HID + tid] = __ldcg(&p.b3[tid]);
    fence_before();
    // after a wait that ran out in an earlier minibatch this one's gradient is not used: it stays zero
    bool ok = __syncthreads_or(failed) == 0;
    fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
    uint32_t phase = 0;
    bool first = true;
    int gi = 0;             // GEMMs issued so far (WaitCfg::skip_gemm)
    bool inflight = false;  // a timed-out wait left MMAs of this CTA pending
    const int ntiles = (n + TILE - 1) / TILE;
    for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int row = tile * TILE + tid;
        const bool valid = row < n;
        float x[IN];
        load_x<false>(X, tile, n, x);
        st_row(sm + O_X, tid, x, IN);
#pragma unroll
        for (int i = 0; i < IN; ++i) st_bf16(sm, O_BT + kmaj(HID + i, tid, TILE), x[i]);
        // ---- layer 1
        ok = gemm(sbase, O_X, O_W1, IN, HID, tmem + C_Z1, false, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        float h1[HID];
        uint64_t m1 = 0;
        for (int c = 0; c < HID; c += 32) tmem_ld32(tmem + lane_base + C_Z1 + c, h1 + c);
#pragma unroll
        for (int j = 0; j < HID; ++j) {
            const float z = h1[j] + sbias[j];
            h1[j] = z > 0.f ? z : 0.f;
            if (z > 0.f) m1 |= (1ull << j);
        }
        st_row(sm + O_H1, tid, h1, HID);
#pragma unroll
        for (int j = 0; j < HID; ++j) st_bf16(sm, O_BT + kmaj(j, tid, TILE), h1[j]);
        // ---- layer 2
        ok = gemm(sbase, O_H1, O_W2, HID, HID, tmem + C_Z2, false, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        float h2[HID];
        uint64_t m2 = 0;
        for (int c = 0; c < HID; c += 32) tmem_ld32(tmem + lane_base + C_Z2 + c, h2 + c);
#pragma unroll
        for (int j = 0; j < HID; ++j) {
            const float z = h2[j] + sbias[HID + j];
            h2[j] = z > 0.f ? z : 0.f;
            if (z > 0.f) m2 |= (1ull << j);
        }
        st_row(sm + O_H2, tid, h2, HID);
#pragma unroll
        for (int j = 0; j < HID; ++j) st_bf16(sm, O_B3 + kmaj(j, tid, TILE), h2[j]);
        // ---- layer 3
        ok = gemm(sbase, O_H2, O_W3, HID, OUT, tmem + C_Y, false, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        float y[OUT];
        tmem_ld16(tmem + lane_base + C_Y, y);
        for (int o = 0; o < OUT; ++o) y[o] += sbias[2 * HID + o];
        // ---- backward
        float dy[OUT];
        float lrow = 0.f;
        for (int o = 0; o < OUT; ++o) dy[o] = 0.f;
        if (valid)
            for (int o = 0; o < USED; ++o) {
                const float e = y[o] - T[2 * (size_t)row + o];
                dy[o] = 2.f * e / (float)n;
                lrow += e * e;
            }
        {
            const float ls = warp_sum(lrow);
            if (lane == 0) swarp[warp][NB] = ls;
        }
        for (int o = 0; o < USED; ++o) {
            const float v = warp_sum(dy[o]);
            if (lane == 0) swarp[warp][2 * HID + o] = v;
        }
        st_row(sm + O_DY, tid, dy, OUT);
        for (int o = 0; o < USED; ++o) st_bf16(sm, O_A3 + kmaj(o, tid, TILE), dy[o]);
        ok = gemm(sbase, O_DY, O_W3T, OUT, HID, tmem + C_Z1, false, mbar, phase, wc, gi, inflight);  // dH2
        if (!ok) break;
        float d2[HID];
        for (int c = 0; c < HID; c += 32) tmem_ld32(tmem + lane_base + C_Z1 + c, d2 + c);
#pragma unroll
        for (int j = 0; j < HID; ++j) {
            d2[j] = ((m2 >> j) & 1ull) ? d2[j] : 0.f;
            st_bf16(sm, O_AT + kmaj(j, tid, TILE), d2[j]);
        }
        st_row(sm + O_DZ2, tid, d2, HID);
#pragma unroll
        for (int c = 0; c < HID; c += 32) {
            const float v = warp_sum32(d2 + c, lane);
            swarp[warp][HID + c + lane] = v;
        }
        ok = gemm(sbase, O_DZ2, O_W2T, HID, HID, tmem + C_Z2, false, mbar, phase, wc, gi, inflight);  // dH1
        if (!ok) break;
        float d1[HID];
        for (int c = 0; c < HID; c += 32) tmem_ld32(tmem + lane_base + C_Z2 + c, d1 + c);
#pragma unroll
        for (int j = 0; j < HID; ++j) {
            d1[j] = ((m1 >> j) & 1ull) ? d1[j] : 0.f;
            st_bf16(sm, O_AT + kmaj(HID + j, tid, TILE), d1[j]);
        }
#pragma unroll
        for (int c = 0; c < HID; c += 32) {
            const float v = warp_sum32(d1 + c, lane);
            swarp[warp][c + lane] = v;
        }
        // this tile's sums, the warps added in order (the tile's other smem
        // writes are fenced by the barrier inside the next GEMM)
        __syncthreads();
        for (int i = tid; i <= NB; i += NT) {
            const float v = ((swarp[0][i] + swarp[1][i]) + swarp[2][i]) + swarp[3][i];
            if (i < NB) sgb[i] += v;
            else sloss += v;
        }
        // weight gradients, accumulated in tensor memory over this CTA's tiles
        ok = gemm(sbase, O_AT, O_BT, TILE, HID + IN, tmem + C_DW12, !first, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        ok = gemm(sbase, O_A3, O_B3, TILE, HID, tmem + C_DW3, !first, mbar, phase, wc, gi, inflight);
        if (!ok) break;
        first = false;
    }
    if (!ok && threadIdx.x == 0) atomicExch(err, 1);
    // MMAs still pending after a timed-out wait write tensor memory: wait for
    // them (bounded again) before that memory is freed below
    if (!ok && inflight) mbar_wait(mbar, phase, kPollLimit);
    {
        // this CTA's part: D12 rows 0..63: dW2 (cols 0..63); rows 64..127:
        // dW1 (cols 64..79); D3 rows 0..15: dW3 (the rows of unused outputs
        // zero); every entry written, zero when the CTA stopped early
        Params g = carve(gpart + (size_t)blockIdx.x * kNParams);
        const bool have = ok && !first;
        const int m = tid;
        float v[16];
        if (m < HID) {
            for (int c = 0; c < HID; c += 16) {
                if (have) tmem_ld16(tmem + lane_base + C_DW12 + c, v);
                for (int i = 0; i < 16; ++i) g.W2[m * HID + c + i] = have ? v[i] : 0.f;
            }
        } else {
            if (have) tmem_ld16(tmem + lane_base + C_DW12 + HID, v);
            for (int i = 0; i < IN; ++i) g.W1[(m - HID) * IN + i] = have ? v[i] : 0.f;
        }
        for (int c = 0; c < HID; c += 16) {
            if (have) tmem_ld16(tmem + lane_base + C_DW3 + c, v);
            if (m < OUT)
                for (int i = 0; i < 16; ++i) g.W3[m * HID + c + i] = (have && m < USED) ? v[i] : 0.f;
        }
        __syncthreads();
        for (int i = tid; i < HID; i += NT) {
            g.b1[i] = have ? sgb[i] : 0.f;
            g.b2[i] = have ? sgb[HID + i] : 0.f;
        }
        if (tid < OUT) g.b3[tid] = have ? sgb[2 * HID + tid] : 0.f;
        if (tid == 0) lpart[blockIdx.x] = have ? (double)sloss / (double)n : 0.0;
    }
    fence_before();
    __syncthreads();
    if (warp == 0) tmem_free<TMEM_COLS>(tmem);
}

// the CTAs' parts of parameter i (or of the loss) added in CTA order
__device__ __forceinline__ float part_sum(const float* part, int nparts, int i) {
    float acc = 0.f;
    int b = 0;
    for (; b + 32 <= nparts; b += 32) {  // (the loads together, the sum in order)
        float v[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __ldcg(&part[(size_t)(b + k) * kNParams + i]);
#pragma unroll
        for (int k = 0; k < 32; ++k) acc += v[k];
    }
    for (; b < nparts; ++b) acc += __ldcg(&part[(size_t)b * kNParams + i]);
    return acc;
}
__device__ __forceinline__ double loss_sum(const double* lpart, int nparts) {
    double l = 0.0;
    int b = 0;
    for (; b + 16 <= nparts; b += 16) {
        double v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = __ldcg(&lpart[b + k]);
#pragma unroll
        for (int k = 0; k < 16; ++k) l += v[k];
    }
    for (; b < nparts; ++b) l += __ldcg(&lpart[b]);
    return l;
}

// g[i] = the CTAs' parts of parameter i; *loss likewise
__global__ void k_grad_sum(const float* __restrict__ part, int nparts, float* g, const double* __restrict__ lpart,
                           double* loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNParams) g[i] = part_sum(part, nparts, i);
    if (i == 0) *loss = loss_sum(lpart, nparts);
}

// What an epoch adds up on the device
struct EpochSum {
    double loss;               // of its minibatches (the gradient call: the loss alone)
    long long steps;           // minibatches applied
};

struct AdamArgs {
    float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ void adam_param(int i, float gi, float* p, float* m, float* v, uint8_t* img, const AdamArgs& a) {
    const float mi = a.b1 * m[i] + (1.f - a.b1) * gi;
    const float vi = a.b2 * v[i] + (1.f - a.b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
    p[i] = pi;
    pack_param(img, i, pi);
}

__global__ void k_adam(float* p, const float* g, float* m, float* v, uint8_t* img, AdamArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNParams) adam_param(i, g[i], p, m, v, img, a);
}

// k_grad_sum and k_adam of one minibatch; the epoch's sums gain it.  After a
// timed-out wait (*err) the network is left as it is.
__global__ void k_grad_adam(const float* part, int nparts, float* g, const double* lpart, EpochSum* sum, float* p,
                            float* m, float* v, uint8_t* img, AdamArgs a, const int* err) {
    pdl_wait();
    pdl_trigger();
    if (__ldcg(err)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNParams) {
        const float gi = part_sum(part, nparts, i);
        g[i] = gi;
        adam_param(i, gi, p, m, v, img, a);
    }
    if (i == 0) {
        sum->loss += loss_sum(lpart, nparts);
        sum->steps += 1;
    }
}

}  // namespace mlp
}  // namespace pgb

struct pg_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    void* memory = nullptr;    // holds all of the below
    float* params = nullptr;   // kNParams
    float* grads = nullptr;
    float* m = nullptr;
    float* v = nullptr;
    uint8_t* img = nullptr;    // BF16 operand images of the weights (P_BYTES), always those of params
    pgb::mlp::EpochSum* sum = nullptr;  // what a training epoch adds up
    float* gpart = nullptr;    // per CTA of a gradient launch: its part of the gradient (kNParams)
    double* lpart = nullptr;   // and of the loss
    int* err = nullptr;
    float* probe = nullptr;    // one tile of inputs and outputs for pg_mlp_wait_selftest
    int step = 0;
    int n_sms = 148;
};

using namespace pgb;
using namespace pgb::mlp;

extern "C" {

int pg_mlp_create(int32_t device, uint64_t seed, pg_mlp** out) {
    if (!out) { set_error("pg_mlp_create: null output"); return PG_ERR_ARG; }
    *out = nullptr;
    pg_mlp* m = new (std::nothrow) pg_mlp;
    if (!m) { set_error("pg_mlp_create: out of host memory"); return PG_ERR_ARG; }
    m->device = device;
    PG_CUDA(cudaSetDevice(device));
    PG_CUDA(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    cudaDeviceGetAttribute(&m->n_sms, cudaDevAttrMultiProcessorCount, device);
    // one allocation, each part on a 256-byte boundary
    struct Part {
        void** p;
        size_t bytes;
    };
    const Part parts[] = {{(void**)&m->params, 4 * (size_t)kNParams * sizeof(float)},
                          {(void**)&m->img, P_BYTES},
                          {(void**)&m->sum, sizeof(EpochSum)},
                          {(void**)&m->err, sizeof(int)},
                          {(void**)&m->probe, TILE * (IN + 2) * sizeof(float)},
                          {(void**)&m->lpart, (size_t)m->n_sms * sizeof(double)},
                          {(void**)&m->gpart, (size_t)m->n_sms * kNParams * sizeof(float)}};
    size_t bytes = 0;
    for (const Part& q : parts) bytes += (q.bytes + 255) & ~size_t(255);
    PG_CUDA(cudaMalloc(&m->memory, bytes));
    PG_CUDA(fill_sync(m->memory, 0, bytes));
    char* at = (char*)m->memory;
    for (const Part& q : parts) {
        *q.p = at;
        at += (q.bytes + 255) & ~size_t(255);
    }
    m->grads = m->params + kNParams;
    m->m = m->grads + kNParams;
    m->v = m->m + kNParams;
    PG_CUDA(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ALLOC));
    for (auto k : {k_mlp_forward<true>, k_mlp_forward<false>})  // room for kForwardCtasPerSm of them on an SM
        PG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    // He initialisation (host, seeded), last layer scaled to start near zero output
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    std::vector<float> h(kNParams, 0.f);
    Params hp = carve(h.data());
    for (int i = 0; i < kW1; ++i) hp.W1[i] = nd(rng) * std::sqrt(2.f / IN);
    for (int i = 0; i < kW2; ++i) hp.W2[i] = nd(rng) * std::sqrt(2.f / HID);
    for (int o = 0; o < USED; ++o)
        for (int j = 0; j < HID; ++j) hp.W3[o * HID + j] = 0.1f * nd(rng) * std::sqrt(1.f / HID);
    PG_CUDA(h2d_sync(m->params, h.data(), kNParams * sizeof(float)));
    k_pack<<<kParamBlocks, 256, 0, m->stream>>>(m->params, m->img);
    PG_CUDA(cudaStreamSynchronize(m->stream));
    *out = m;
    return PG_OK;
}

void pg_mlp_destroy(pg_mlp* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    if (m->memory) cudaFree(m->memory);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
}

int32_t pg_mlp_param_count(void) { return kNParams; }

int pg_mlp_params(pg_mlp* m, float* host, int32_t set) {
    if (!m || !host) { set_error("pg_mlp_params: null argument"); return PG_ERR_ARG; }
    cudaSetDevice(m->device);
    PG_CUDA(cudaStreamSynchronize(m->stream));
    if (set) {
        PG_CUDA(h2d_sync(m->params, host, kNParams * sizeof(float)));
        PG_CUDA(fill_sync(m->m, 0, 2 * kNParams * sizeof(float)));
        k_pack<<<kParamBlocks, 256, 0, m->stream>>>(m->params, m->img);
        PG_CUDA(cudaStreamSynchronize(m->stream));  // a forward pass may follow on another stream
        m->step = 0;
    } else {
        PG_CUDA(cudaMemcpy(host, m->params, kNParams * sizeof(float), cudaMemcpyDeviceToHost));
    }
    return PG_OK;
}

int pg_mlp_grads(pg_mlp* m, float* host) {
    if (!m || !host) { set_error("pg_mlp_grads: null argument"); return PG_ERR_ARG; }
    cudaSetDevice(m->device);
    PG_CUDA(cudaStreamSynchronize(m->stream));
    PG_CUDA(cudaMemcpy(host, m->grads, kNParams * sizeof(float), cudaMemcpyDeviceToHost));
    return PG_OK;
}

static int mlp_check_err(pg_mlp* m) {
    int e = 0;
    PG_CUDA(cudaMemcpyAsync(&e, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    PG_CUDA(cudaStreamSynchronize(m->stream));
    if (e) {
        cudaMemsetAsync(m->err, 0, sizeof(int), m->stream);
        set_error("pg_mlp: tensor-core completion wait timed out");
        return PG_ERR_STATE;
    }
    return PG_OK;
}

static void launch_forward(pg_mlp* m, const float* X, int n, float* Y, cudaStream_t s, WaitCfg wc) {
    const int tiles = (n + TILE - 1) / TILE, grid = std::min(tiles, m->n_sms * kForwardCtasPerSm);
    const Params p = carve(m->params);
    const uint4* img = reinterpret_cast<const uint4*>(m->img);
    // 16-byte loads of X and 8-byte stores of Y where the caller's buffers are so aligned
    const bool vec = (reinterpret_cast<uintptr_t>(X) & 15) == 0 && (reinterpret_cast<uintptr_t>(Y) & 7) == 0;
    if (vec) k_mlp_forward<true><<<grid, NT, F_ALLOC, s>>>(X, n, p, img, Y, m->err, wc);
    else k_mlp_forward<false><<<grid, NT, F_ALLOC, s>>>(X, n, p, img, Y, m->err, wc);
}

// Y_dev[2n] = MLP(X_dev[16n]) (device pointers)
int pg_mlp_forward(pg_mlp* m, const float* X_dev, int32_t n, float* Y_dev, void* stream) {
    if (!m || (n > 0 && (!X_dev || !Y_dev))) { set_error("pg_mlp_forward: null argument"); return PG_ERR_ARG; }
    if (n <= 0) return PG_OK;
    cudaSetDevice(m->device);
    cudaStream_t s = stream ? (cudaStream_t)stream : m->stream;
    launch_forward(m, X_dev, n, Y_dev, s, WaitCfg{kPollLimit, -1});
    PG_CUDA(cudaGetLastError());
    if (s == m->stream) return mlp_check_err(m);
    return PG_OK;
}

// the CTAs' gradient parts over n rows; returns their number
static int launch_train(pg_mlp* m, const float* X, const float* T, int n, WaitCfg wc) {
    const int tiles = (n + TILE - 1) / TILE, grid = std::min(tiles, m->n_sms);
    launch_pdl(k_mlp_train, grid, NT, SMEM_ALLOC, m->stream, X, T, n, carve(m->params),
               reinterpret_cast<const uint4*>(m->img), m->gpart, m->lpart, m->err, wc);
    return grid;
}

// Adam's constants of the next step
static AdamArgs next_step(pg_mlp* m, float lr) {
    m->step += 1;
    AdamArgs a;
    a.lr = lr;
    a.b1 = 0.9f;
    a.b2 = 0.999f;
    a.eps = 1e-8f;
    a.c1 = 1.f - std::pow(a.b1, (float)m->step);
    a.c2 = 1.f - std::pow(a.b2, (float)m->step);
    return a;
}

// gradients of the mean-squared loss over all n rows into the internal buffer; loss to *loss_host
int pg_mlp_gradient(pg_mlp* m, const float* X_dev, const float* T_dev, int32_t n, double* loss_host) {
    if (!m || !X_dev || !T_dev || n <= 0) { set_error("pg_mlp_gradient: bad argument"); return PG_ERR_ARG; }
    cudaSetDevice(m->device);
    const int parts = launch_train(m, X_dev, T_dev, n, WaitCfg{kPollLimit, -1});
    PG_CUDA(cudaGetLastError());
    k_grad_sum<<<kParamBlocks, 256, 0, m->stream>>>(m->gpart, parts, m->grads, m->lpart, &m->sum->loss);
    PG_CUDA(cudaGetLastError());
    int rc = mlp_check_err(m);
    if (rc) return rc;
    if (loss_host) PG_CUDA(cudaMemcpy(loss_host, &m->sum->loss, sizeof(double), cudaMemcpyDeviceToHost));
    return PG_OK;
}

int pg_mlp_adam(pg_mlp* m, float lr) {
    if (!m) { set_error("pg_mlp_adam: null"); return PG_ERR_ARG; }
    cudaSetDevice(m->device);
    k_adam<<<kParamBlocks, 256, 0, m->stream>>>(m->params, m->grads, m->m, m->v, m->img, next_step(m, lr));
    PG_CUDA(cudaGetLastError());
    return PG_OK;
}

// One pass over n rows in batches of `batch` rows, queued whole: the host
// looks at its loss and at the error word once, at its end.  A minibatch whose
// wait ran out and those after it are not applied, and not counted as steps.
// `first` is the first minibatch's WaitCfg.
static int train_epoch(pg_mlp* m, const float* X, const float* T, int n, int batch, float lr, WaitCfg first, double* loss) {
    PG_CUDA(cudaMemsetAsync(m->sum, 0, sizeof(EpochSum), m->stream));
    const int step0 = m->step;
    int nb = 0;
    for (int s0 = 0; s0 < n; s0 += batch) {
        const int nn = (n - s0) < batch ? (n - s0) : batch;
        const int parts = launch_train(m, X + (size_t)s0 * IN, T + (size_t)s0 * 2, nn, nb ? WaitCfg{kPollLimit, -1} : first);
        launch_pdl(k_grad_adam, kParamBlocks, 256, 0, m->stream, m->gpart, parts, m->grads, m->lpart, m->sum,
                   m->params, m->m, m->v, m->img, next_step(m, lr), m->err);
        PG_CUDA(cudaGetLastError());
        ++nb;
    }
    EpochSum sum{};
    PG_CUDA(cudaMemcpyAsync(&sum, m->sum, sizeof sum, cudaMemcpyDeviceToHost, m->stream));
    const int rc = mlp_check_err(m);
    if (rc) {
        m->step = step0 + (int)sum.steps;
        return rc;
    }
    if (loss) *loss = sum.loss / (nb ? nb : 1);
    return PG_OK;
}

// Minibatch training: `epochs` passes over n rows in batches of `batch` rows
// (the caller shuffles).  Writes the mean loss of every epoch to loss_hist.
int pg_mlp_train(pg_mlp* m, const float* X_dev, const float* T_dev, int32_t n, int32_t epochs, int32_t batch, float lr,
                 double* loss_hist) {
    if (!m || !X_dev || !T_dev || n <= 0 || batch <= 0) { set_error("pg_mlp_train: bad argument"); return PG_ERR_ARG; }
    cudaSetDevice(m->device);
    for (int ep = 0; ep < epochs; ++ep) {
        const int rc = train_epoch(m, X_dev, T_dev, n, batch, lr, WaitCfg{kPollLimit, -1}, loss_hist ? loss_hist + ep : nullptr);
        if (rc) return rc;
    }
    return PG_OK;
}

// Self-test of the bounded completion wait: one forward tile, and an epoch of
// two minibatches, whose first GEMM is not issued, so nothing arrives on its
// mbarrier and the wait must give up after `polls` polls.  Nothing is in
// flight when it does, so the kernel records its error word, frees its tensor
// memory and returns; the call returns the timeout status, and the network is
// what it was.
int pg_mlp_wait_selftest(pg_mlp* m, int32_t polls) {
    if (!m || polls < 1) { set_error("pg_mlp_wait_selftest: bad argument"); return PG_ERR_ARG; }
    cudaSetDevice(m->device);
    launch_forward(m, m->probe, TILE, m->probe + TILE * IN, m->stream, WaitCfg{polls, 0});
    PG_CUDA(cudaGetLastError());
    const int rc = mlp_check_err(m);
    if (rc != PG_ERR_STATE) return rc;
    return train_epoch(m, m->probe, m->probe + TILE * IN, TILE, TILE / 2, 1e-3f, WaitCfg{polls, 0}, nullptr);
}

}  // extern "C"
