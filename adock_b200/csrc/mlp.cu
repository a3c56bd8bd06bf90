// Proposal network kernels (sm_100a): BF16 GEMM on the tensor cores with FP32 accumulation and fused epilogues,
// Gaussian negative log-likelihood + its gradient, SiLU backward, bias-gradient reduction, Adam.
//
// Network: x [320] -> SiLU(W1 x + b1) [256] -> SiLU(W2 h1 + b2) [256] -> W3 h2 + b3 [64]. Output columns 0..25 are
// the means and 32..57 the log standard deviations of the move (translation 3, rotation vector 3, torsions 20);
// with a translation mixture, columns 27..29 and 58..60 hold two more translation means and 26, 30, 61 the
// mixing logits.
//
// GEMM: C[M,N] = A[M,K] B[K,N] with A and B in BF16 at arbitrary (row, column) strides, so the same kernel serves
// the forward pass (X W), the input gradient (dY W^T) and the weight gradient (X^T dY). adock_gemm_bf16 runs it on
// the tcgen05 tensor cores with the accumulator in tensor memory (gemm_bf16_tc_kernel); gemm_bf16_kernel is an
// independent warp-level mma.sync version (64x64 CTA tile, 4 warps of 32x32, K step 32, m16n8k16 BF16 -> FP32)
// behind adock_gemm_bf16_mma, which the tests use as a cross-check.
//
// adock_mlp_forward and adock_mlp_loss_grad queue a whole forward pass, or forward and backward pass, from one call:
// the layers are a few microseconds each, so the launches' host cost would otherwise decide.
#include "common.cuh"
#include "mma_ring.h"

namespace adock {

#define GM 64
#define GN 64
#define GK 32
#define APAD 8

struct GemmArgs {
    int M, N, K;
    const __nv_bfloat16* A;
    long long sAm, sAk;
    const __nv_bfloat16* B;
    long long sBk, sBn;
    // epilogue
    float* C;             // FP32 output [M, ldc] (optional)
    long long ldc;
    float beta;           // C = acc + beta * C
    const float* bias;    // [N] (optional)
    int act;              // 0 none, 1 SiLU
    float* pre;           // FP32 pre-activation copy [M, ldc] (optional)
    __nv_bfloat16* Cb;    // BF16 output [M, ldcb] (optional)
    long long ldcb;
    const float* dpre;    // with it, C is multiplied by SiLU'(dpre) ([M, ldcb], tcgen05 kernel only)
    int vec;              // rows of C, pre, Cb, dpre and bias can be read and written 4 columns at a time
};

__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }

__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__global__ void __launch_bounds__(128) gemm_bf16_kernel(const __grid_constant__ GemmArgs g) {
    __shared__ __align__(16) __nv_bfloat16 As[GM][GK + APAD];   // [m][k]
    __shared__ __align__(16) __nv_bfloat16 Bs[GN][GK + APAD];   // [n][k] (transposed: k contiguous)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GN;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int gid = lane >> 2, tig = lane & 3;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.f;
    const bool a_kfast = g.sAk == 1, b_kfast = g.sBk == 1;
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    for (int k0 = 0; k0 < g.K; k0 += GK) {
        // stage A[m0:m0+64, k0:k0+32] and B[k0:k0+32, n0:n0+64]; the contiguous dimension runs across threads
        for (int e = tid; e < GM * GK; e += 128) {
            const int mm = a_kfast ? e / GK : e % GM, kk = a_kfast ? e % GK : e / GM;
            const int m = m0 + mm, k = k0 + kk;
            As[mm][kk] = (m < g.M && k < g.K) ? g.A[(long long)m * g.sAm + (long long)k * g.sAk] : zero;
        }
        for (int e = tid; e < GN * GK; e += 128) {
            const int nn = b_kfast ? e / GK : e % GN, kk = b_kfast ? e % GK : e / GN;
            const int n = n0 + nn, k = k0 + kk;
            Bs[nn][kk] = (n < g.N && k < g.K) ? g.B[(long long)k * g.sBk + (long long)n * g.sBn] : zero;
        }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < GK; ks += 16) {
            uint32_t af[2][4], bf[4][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = wm + i * 16 + gid;
                af[i][0] = *(const uint32_t*)&As[r][ks + tig * 2];
                af[i][1] = *(const uint32_t*)&As[r + 8][ks + tig * 2];
                af[i][2] = *(const uint32_t*)&As[r][ks + tig * 2 + 8];
                af[i][3] = *(const uint32_t*)&As[r + 8][ks + tig * 2 + 8];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = wn + j * 8 + gid;
                bf[j][0] = *(const uint32_t*)&Bs[c][ks + tig * 2];
                bf[j][1] = *(const uint32_t*)&Bs[c][ks + tig * 2 + 8];
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], af[i], bf[j]);
        }
        __syncthreads();
    }
    // epilogue: acc[i][j] = rows (gid, gid + 8), cols (tig * 2, tig * 2 + 1) of tile (i, j)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int m = m0 + wm + i * 16 + gid + (r >> 1) * 8;
                const int n = n0 + wn + j * 8 + tig * 2 + (r & 1);
                if (m >= g.M || n >= g.N) continue;
                float v = acc[i][j][r];
                if (g.C && g.beta != 0.f) v += g.beta * g.C[(long long)m * g.ldc + n];
                if (g.bias) v += g.bias[n];
                if (g.pre) g.pre[(long long)m * g.ldc + n] = v;
                if (g.act == 1) v = silu(v);
                if (g.C) g.C[(long long)m * g.ldc + n] = v;
                if (g.Cb) g.Cb[(long long)m * g.ldcb + n] = __float2bfloat16(v);
            }
}

// ------------------------------------------------------------------------------------------------ tcgen05 GEMM
// Same product and epilogue on the 5th-generation tensor cores. One CTA of 256 threads computes a 128 x TN tile
// (TN = 64 or 128) of C with the FP32 accumulator in tensor memory (TMEM: 128 lanes = rows, TN columns):
//  - K is stepped by 64 through a ring of TC_STAGES shared-memory stages. The threads load A[128, 64] and B[64, TN] of
//    the next step into registers while the tensor core works on the current one, then write them in the canonical
//    K-major layout without swizzle: 8-row x 16-byte core matrices, core matrix (row group g, K chunk c) at byte
//    g * TC_SBO + c * 128, row r of it at + 16 r. B is stored as its transpose (TN rows of K), so the MMA computes
//    D[m, n] = sum_k A[m, k] B^T[n, k]. TC_SBO is 1,040 and not 1,024 so that eight row groups start in different banks.
//    An operand whose K or row dimension is contiguous and 16-byte aligned is read in 16-byte vectors (a contiguous row
//    dimension in 8 x 8 blocks that are transposed in registers); any other strides element by element.
//  - After a proxy fence and a CTA barrier, one thread issues four tcgen05.mma (M 128, N TN, K 16; BF16 inputs,
//    FP32 accumulate; descriptor start address advanced by two core matrices per MMA, leading byte offset 128 =
//    the next K chunk, stride byte offset TC_SBO = the next row group) and tcgen05.commit, which arrives on the
//    stage's mbarrier when they have completed; a stage is refilled after its barrier.
//  - Few tiles over a long K (the weight gradients: K = batch) would leave most SMs idle: a cluster of up to 8 CTAs
//    then splits K of one tile. Each leaves its partial tile in shared memory and sums one slice of rows over the
//    cluster's CTAs, always in rank order.
//  - Epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 (its 32 rows) and half the columns, 16 at a time with
//    tcgen05.ld, and applies C = acc + beta C + bias, pre-activation copy, SiLU, FP32 and BF16 stores.
// Every mbarrier wait is bounded; a wait that gives up sets g_tc_status (read by adock_gemm_status) and the cluster
// skips the rest of its tile, then frees its TMEM.
// Bound by the latency of the loads at these sizes (4-8 K steps per CTA). Before (one stage, element loads, no split)
// the three layers of 8,192 rows took 422 us and the weight gradient 320 x 256 over 4,096 rows 2.9 ms on 6 CTAs; now
// 49 us and 17 us.
#define TC_BM 128
#define TC_BK 64
#define TC_STAGES 3
#define TC_SBO 1040
#define TC_THREADS 256
#define TC_WAIT_MAX (1 << 22)
#define TC_WAIT_NS 200000000ull   // 200 ms

__device__ int g_tc_status;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start address, leading / stride byte offsets (all >> 4), version 1 at bit 46,
// base offset 0, layout type 0 (no swizzle) at bits 61..63.
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator (bit 4), A and B BF16 (bits 7 and 10), both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for the mbarrier phase of the given parity; gives up after TC_WAIT_MAX polls or TC_WAIT_NS nanoseconds of
// the global timer, whichever comes first (a poll may suspend the thread for a system-dependent time).
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity) {
    const uint64_t t0 = global_ns();
    for (int i = 0; i < TC_WAIT_MAX; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if (global_ns() - t0 > TC_WAIT_NS) return false;
    }
    return false;
}

// How the staging reads an operand: 16-byte vectors along K, 16-byte vectors along its rows (A's M, B's N), elements.
enum { OP_KVEC, OP_ROWVEC, OP_ELEM };

// One operand's K step (ROWS rows x 64 K) on its way through registers.
template <int ROWS>
struct Operand {
    static constexpr int VEC = ROWS * 8 / TC_THREADS;   // K vectors per thread
    static constexpr int BLK = ROWS;                    // 8 x 8 blocks
    uint4 r[8];

    // first: first thread of the block loads (the two operands of a step use different threads)
    __device__ __forceinline__ void load(const __nv_bfloat16* X, long long s_row, long long s_k, int row0, int rows, int k0,
                                         int K, int mode, int first) {
        const uint4 zero = make_uint4(0, 0, 0, 0);
        if (mode == OP_KVEC) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
                const int t = threadIdx.x + v * TC_THREADS;
                const int row = row0 + (t >> 6) * 8 + (t & 7), k = k0 + ((t >> 3) & 7) * 8;
                r[v] = row < rows && k < K ? __ldg((const uint4*)(X + row * s_row + k)) : zero;
            }
        } else if (mode == OP_ROWVEC) {
            const int t = (int)threadIdx.x - first;
            if (t >= 0 && t < BLK) {
                const int row = row0 + (t % (ROWS / 8)) * 8, k = k0 + (t / (ROWS / 8)) * 8;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    r[j] = row < rows && k + j < K ? __ldg((const uint4*)(X + (k + j) * s_k + row)) : zero;
            }
        }
    }

    __device__ __forceinline__ void store(unsigned char* S, const __nv_bfloat16* X, long long s_row, long long s_k, int row0,
                                          int rows, int k0, int K, int mode, int first) const {
        if (mode == OP_KVEC) {
#pragma unroll
            for (int v = 0; v < VEC; ++v) {
                const int t = threadIdx.x + v * TC_THREADS;
                *(uint4*)(S + (t >> 6) * TC_SBO + ((t >> 3) & 7) * 128 + (t & 7) * 16) = r[v];
            }
        } else if (mode == OP_ROWVEC) {
            const int t = (int)threadIdx.x - first;
            if (t >= 0 && t < BLK) {
                unsigned char* d = S + (t % (ROWS / 8)) * TC_SBO + (t / (ROWS / 8)) * 128;
#pragma unroll
                for (int e = 0; e < 8; ++e) {   // row e of the block: element e of the eight vectors
                    const uint32_t sel = (e & 1) ? 0x7632u : 0x5410u;
                    uint32_t w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) w[q] = __byte_perm(word(r[2 * q], e >> 1), word(r[2 * q + 1], e >> 1), sel);
                    *(uint4*)(d + e * 16) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        } else {
            const bool k_fast = s_k == 1;
            for (int e = threadIdx.x; e < ROWS * TC_BK; e += TC_THREADS) {
                const int row = k_fast ? e / TC_BK : e % ROWS, k = k_fast ? e % TC_BK : e / ROWS;
                const __nv_bfloat16 v = row0 + row < rows && k0 + k < K ? X[(row0 + row) * s_row + (k0 + k) * s_k]
                                                                        : __float2bfloat16(0.f);
                *(__nv_bfloat16*)(S + (row >> 3) * TC_SBO + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2) = v;
            }
        }
    }

    static __device__ __forceinline__ uint32_t word(const uint4& v, int i) {
        return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
    }
};

// d * SiLU'(a)
__device__ __forceinline__ float silu_back(float d, float a) {
    const float s = 1.f / (1.f + __expf(-a));
    return d * s * (1.f + a * (1.f - s));
}

// Epilogue of four columns n..n+3 of row m.
__device__ __forceinline__ void tc_epilogue(const GemmArgs& g, int m, int n, const float* acc) {
    const long long c = (long long)m * g.ldc + n, cb = (long long)m * g.ldcb + n;
    if (g.vec && n + 4 <= g.N) {
        float4 v = make_float4(acc[0], acc[1], acc[2], acc[3]);
        if (g.C && g.beta != 0.f) {
            const float4 o = *(const float4*)(g.C + c);
            v.x += g.beta * o.x; v.y += g.beta * o.y; v.z += g.beta * o.z; v.w += g.beta * o.w;
        }
        if (g.bias) {
            const float4 o = *(const float4*)(g.bias + n);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        if (g.pre) *(float4*)(g.pre + c) = v;
        if (g.act == 1) { v.x = silu(v.x); v.y = silu(v.y); v.z = silu(v.z); v.w = silu(v.w); }
        if (g.dpre) {
            const float4 a = *(const float4*)(g.dpre + cb);
            v.x = silu_back(v.x, a.x); v.y = silu_back(v.y, a.y); v.z = silu_back(v.z, a.z); v.w = silu_back(v.w, a.w);
        }
        if (g.C) *(float4*)(g.C + c) = v;
        if (g.Cb) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
            *(uint2*)(g.Cb + cb) = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
        }
        return;
    }
    for (int j = 0; j < 4 && n + j < g.N; ++j) {
        float v = acc[j];
        if (g.C && g.beta != 0.f) v += g.beta * g.C[c + j];
        if (g.bias) v += g.bias[n + j];
        if (g.pre) g.pre[c + j] = v;
        if (g.act == 1) v = silu(v);
        if (g.dpre) v = silu_back(v, g.dpre[cb + j]);
        if (g.C) g.C[c + j] = v;
        if (g.Cb) g.Cb[cb + j] = __float2bfloat16(v);
    }
}

// The .aligned instructions below (cluster barriers, tcgen05 allocation and loads) need all lanes of a warp together; after a
// branch or loop that lanes leave apart a __syncwarp() makes that certain.
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int TN>
struct TcSmem {
    static constexpr int A = TC_BM / 8 * TC_SBO, B = TN / 8 * TC_SBO, STAGE = A + B;
    static constexpr int ROW = TN + 4;   // floats per row of a partial tile (conflict-free 16-byte writes)
    static constexpr int TOTAL = TC_STAGES * STAGE;
    static_assert(TC_BM * ROW * 4 <= TOTAL, "the partial tile reuses the stages");
};

// gridDim.z = the cluster's CTAs along K (1: no cluster)
template <int TN>
__global__ void __launch_bounds__(TC_THREADS, 2) gemm_bf16_tc_kernel(const __grid_constant__ GemmArgs g, int a_mode,
                                                                     int b_mode) {
    extern __shared__ __align__(16) unsigned char tc_smem[];
    using SM = TcSmem<TN>;
    __shared__ __align__(8) uint64_t mbar[TC_STAGES];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int fail_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * TN;
    const int split = gridDim.z, rank = blockIdx.z;
    if (tid == 0) {
        fail_sh = 0;
        for (int s = 0; s < TC_STAGES; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar[s])), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_sh)), "r"(TN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_sh;
    const int nk = (g.K + TC_BK - 1) / TC_BK;
    const int k_begin = (int)((long long)nk * rank / split), k_end = (int)((long long)nk * (rank + 1) / split);
    const int steps = k_end - k_begin;
    Operand<TC_BM> a;
    Operand<TN> b;
    auto load = [&](int kt) {
        a.load(g.A, g.sAm, g.sAk, m0, g.M, kt * TC_BK, g.K, a_mode, 0);
        b.load(g.B, g.sBn, g.sBk, n0, g.N, kt * TC_BK, g.K, b_mode, TC_THREADS / 2);
    };
    if (steps > 0) load(k_begin);
    auto wait = [&](int s, unsigned parity) { return tc_wait(smem_u32(&mbar[s]), parity); };
    auto fill = [&](int it, int s) {
        const int k0 = (k_begin + it) * TC_BK;
        unsigned char* As = tc_smem + s * SM::STAGE;
        a.store(As, g.A, g.sAm, g.sAk, m0, g.M, k0, g.K, a_mode, 0);
        b.store(As + SM::A, g.B, g.sBn, g.sBk, n0, g.N, k0, g.K, b_mode, TC_THREADS / 2);
        if (it + 1 < steps) load(k_begin + it + 1);
        // make the generic-proxy stores visible to the tensor core (async proxy) before the barrier
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    };
    auto any = [&](bool flag) { return __syncthreads_or(flag) != 0; };
    auto issue = [&](int it, int s) {
        if (tid != 0) return;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = smem_u32(tc_smem + s * SM::STAGE), b0 = a0 + SM::A;
#pragma unroll
        for (int q = 0; q < TC_BK / 16; ++q) {
            const uint64_t da = tc_smem_desc(a0 + q * 256, 128, TC_SBO);
            const uint64_t db = tc_smem_desc(b0 + q * 256, 128, TC_SBO);
            const uint32_t acc = (it > 0 || q > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                ::"r"(tmem), "l"(da), "l"(db), "r"(tc_idesc(TC_BM, TN)), "r"(acc)
                : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                     ::"r"(smem_u32(&mbar[s])) : "memory");
    };
    // after a wait that gave up the tile is not written: its MMAs may be incomplete, and where the last wait gave up too,
    // still read the stages that the partial tile would overwrite
    const bool ok = run_ring<TC_STAGES>(steps, wait, fill, any, issue);
    if (tid == 0 && !ok) {
        fail_sh = 1;   // for the cluster, which reads it after its barrier
        atomicExch(&g_tc_status, 1);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int row = (warp & 3) * 32 + lane, c_begin = (warp >> 2) * (TN / 2);
    float* part = (float*)tc_smem;
    if (ok) {
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_begin + TN / 2; c0 += 16) {
            uint32_t r[16];
            __syncwarp();
            if (steps > 0) {
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15])
                    : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            } else {   // K = 0: the product is zero; only the epilogue terms remain
#pragma unroll
                for (int j = 0; j < 16; ++j) r[j] = 0u;
            }
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                const float v[4] = {__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                    __uint_as_float(r[j + 3])};
                if (split > 1) *(float4*)(part + row * SM::ROW + c0 + j) = make_float4(v[0], v[1], v[2], v[3]);
                else if (m0 + row < g.M) tc_epilogue(g, m0 + row, n0 + c0 + j, v);
            }
        }
    }
    if (split > 1) {
        cluster_sync();
        uint32_t peer[8];
        int failed = 0;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const uint32_t q = (uint32_t)(p < split ? p : 0);
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer[p]) : "r"(smem_u32(part)), "r"(q));
            uint32_t f;
            int v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(f) : "r"(smem_u32(&fail_sh)), "r"(q));
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(f) : "memory");
            failed |= v;
        }
        const int r_begin = TC_BM * rank / split, r_end = TC_BM * (rank + 1) / split;
        if (!failed)
            for (int t = tid; t < (r_end - r_begin) * (TN / 4); t += TC_THREADS) {
                const int rr = r_begin + t / (TN / 4), cc = (t % (TN / 4)) * 4;
                if (m0 + rr >= g.M) break;
                float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    if (p >= split) break;
                    float4 o;
                    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                                 : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w)
                                 : "r"(peer[p] + (uint32_t)((rr * SM::ROW + cc) * 4)) : "memory");
                    v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
                }
                tc_epilogue(g, m0 + rr, n0 + cc, v);
            }
        cluster_sync();   // the peers' partial tiles stay until everyone has read them
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN) : "memory");
    }
}

// Gaussian NLL over the move dimensions: out [B, 64] (mu = out[:, 0:26], log_sigma = out[:, 32:58] clamped to
// [-4, 2]); target [B, 32] (move in 0..25, torsion count in 26); rows of the batch weighted equally.
// n_comp = 3: the translation is a mixture of 3 Gaussians with the shared per-axis sigma (out[:, 32:35]), means at
// columns 0, 27, 58 (3 each) and mixing logits at columns 26, 30, 61; its term is
// -log sum_k softmax(logits)_k N(t | mu_k, sigma). Rotation and torsions stay single Gaussians.
// Writes dOut (BF16, [B, 64]) = d(mean loss)/d(out) and accumulates the loss sum into *loss (one atomic per block: one
// per row queued up at the single address).
#define NLL_WARPS 8
__constant__ int MIX_MEAN[3] = {0, 27, 58};
__constant__ int MIX_LOGIT[3] = {26, 30, 61};

__global__ void nll_kernel(const float* __restrict__ out, const float* __restrict__ target, int B, int n_comp,
                           __nv_bfloat16* __restrict__ dout, float* __restrict__ loss) {
    __shared__ float part[NLL_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float sum = 0.f;
    for (int row = blockIdx.x * NLL_WARPS + warp; row < B; row += gridDim.x * NLL_WARPS) {
        const float* o = out + (long long)row * 64;
        const float* t = target + (long long)row * 32;
        const int nt = (int)t[26];
        const float inv = 1.f / (float)B;
        const bool mix = n_comp > 1;
        float l = 0.f, dmu = 0.f, dls = 0.f;
        const int d = lane;
        const bool active = d < 26 && (d < 6 || d - 6 < nt) && !(mix && d < 3);
        if (active) {
            const float mu = o[d], ls_raw = o[32 + d];
            const float ls = fminf(fmaxf(ls_raw, -4.f), 2.f);
            const float z = (t[d] - mu) * __expf(-ls);
            l = 0.5f * z * z + ls;
            dmu = -z * __expf(-ls) * inv;
            dls = (ls_raw > -4.f && ls_raw < 2.f) ? (1.f - z * z) * inv : 0.f;
        }
        dout[(long long)row * 64 + lane] = __float2bfloat16(dmu);
        dout[(long long)row * 64 + 32 + lane] = __float2bfloat16(dls);
        if (mix) {
            __syncwarp();
            if (lane == 0) {   // the translation mixture: overwrites its columns after the per-lane defaults (0)
                float ls[3], isd[3], lg[3], lp[3], z[3][3];
                for (int a = 0; a < 3; ++a) {
                    ls[a] = fminf(fmaxf(o[32 + a], -4.f), 2.f);
                    isd[a] = __expf(-ls[a]);
                }
                float mg = -3.4e38f, mp = -3.4e38f;
                for (int k = 0; k < 3; ++k) {
                    lg[k] = o[MIX_LOGIT[k]];
                    lp[k] = lg[k];
                    for (int a = 0; a < 3; ++a) {
                        z[k][a] = (t[a] - o[MIX_MEAN[k] + a]) * isd[a];
                        lp[k] -= 0.5f * z[k][a] * z[k][a];
                    }
                    mg = fmaxf(mg, lg[k]);
                    mp = fmaxf(mp, lp[k]);
                }
                float sg = 0.f, sp = 0.f;
                for (int k = 0; k < 3; ++k) {
                    sg += __expf(lg[k] - mg);
                    sp += __expf(lp[k] - mp);
                }
                const float lse_g = mg + __logf(sg), lse_p = mp + __logf(sp);
                l += lse_g - lse_p + ls[0] + ls[1] + ls[2];
                float dl[3] = {0.f, 0.f, 0.f};
                for (int k = 0; k < 3; ++k) {
                    const float r = __expf(lp[k] - lse_p), p = __expf(lg[k] - lse_g);
                    dout[(long long)row * 64 + MIX_LOGIT[k]] = __float2bfloat16((p - r) * inv);
                    for (int a = 0; a < 3; ++a) {
                        dout[(long long)row * 64 + MIX_MEAN[k] + a] = __float2bfloat16(-r * z[k][a] * isd[a] * inv);
                        dl[a] += r * (1.f - z[k][a] * z[k][a]);
                    }
                }
                for (int a = 0; a < 3; ++a) {
                    const float raw = o[32 + a];
                    dout[(long long)row * 64 + 32 + a] = __float2bfloat16((raw > -4.f && raw < 2.f) ? dl[a] * inv : 0.f);
                }
            }
        }
        sum += l;
    }
    sum = warp_sum(sum);
    if (lane == 0) part[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < NLL_WARPS; ++w) t += part[w];
        atomicAdd(loss, t);
    }
}

// dA = dH * SiLU'(A) (A = pre-activation FP32), BF16 output
__global__ void silu_backward_kernel(const float* __restrict__ dH, const float* __restrict__ A, long long n,
                                     __nv_bfloat16* __restrict__ dA) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        dA[i] = __float2bfloat16(silu_back(dH[i], A[i]));
    }
}

// db[n] = sum_rows dA[row, n] (BF16 input, FP32 sums). A cluster of BIAS_SPLIT blocks shares 64 columns: each block
// sums a range of rows, 8 columns (one 16-byte vector where `vec`) per thread and 32 rows at a time; the first block adds
// the others' sums in rank order. (One block per 32 columns with 2-byte loads left 140 SMs idle: 54 us for 4,096 x 256,
// now 8 us.)
#define BIAS_SPLIT 8
__global__ void __launch_bounds__(256) __cluster_dims__(1, BIAS_SPLIT, 1)
    bias_grad_kernel(const __nv_bfloat16* __restrict__ dA, int rows, int cols, int vec, float* __restrict__ db) {
    __shared__ float part[32][65];
    __shared__ float total[64];
    const int c8 = threadIdx.x & 7, line = threadIdx.x >> 3, rank = blockIdx.y;
    const int c0 = blockIdx.x * 64 + c8 * 8;
    const int r_begin = (int)((long long)rows * rank / BIAS_SPLIT), r_end = (int)((long long)rows * (rank + 1) / BIAS_SPLIT);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (vec) {
        if (c0 < cols) {
#pragma unroll 4
            for (int r = r_begin + line; r < r_end; r += 32) {
                const uint4 v = __ldg((const uint4*)(dA + (long long)r * cols + c0));
                const __nv_bfloat162* h = (const __nv_bfloat162*)&v;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __bfloat1622float2(h[j]);
                    s[2 * j] += f.x;
                    s[2 * j + 1] += f.y;
                }
            }
        }
    } else {
        for (int r = r_begin + line; r < r_end; r += 32)
            for (int j = 0; j < 8; ++j)
                if (c0 + j < cols) s[j] += __bfloat162float(dA[(long long)r * cols + c0 + j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) part[line][c8 * 8 + j] = s[j];
    __syncthreads();
    if (threadIdx.x < 64) {
        float t = 0.f;
        for (int i = 0; i < 32; ++i) t += part[i][threadIdx.x];
        total[threadIdx.x] = t;
    }
    cluster_sync();
    const int c = blockIdx.x * 64 + threadIdx.x;
    if (rank == 0 && threadIdx.x < 64 && c < cols) {
        float t = 0.f;
        for (int p = 0; p < BIAS_SPLIT; ++p) {
            uint32_t at;
            float v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(&total[threadIdx.x])), "r"(p));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
            t += v;
        }
        db[c] = t;
    }
    cluster_sync();
}

// Adam on FP32 master parameters, refreshing their BF16 copies (bias_hat corrections from the step count)
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ grad, float* __restrict__ m,
                            float* __restrict__ v, __nv_bfloat16* __restrict__ pb, long long n, float lr, float b1,
                            float b2, float eps, float c1, float c2, float wd) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = grad[i] + wd * p[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        if (pb) pb[i] = __float2bfloat16(pi);
    }
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16(x[i]);
}

static void launch_nll(const float* out, const float* target, int B, int n_comp, __nv_bfloat16* dout, float* loss,
                       cudaStream_t st) {
    const int blocks = min((B + NLL_WARPS - 1) / NLL_WARPS, sm_count() * 4);
    nll_kernel<<<blocks, 32 * NLL_WARPS, 0, st>>>(out, target, B, n_comp, dout, loss);
}

static int launch_bias_grad(const __nv_bfloat16* dA, int rows, int cols, float* db, cudaStream_t st) {
    const int vec = cols % 8 == 0 && ((uintptr_t)dA & 15) == 0;
    bias_grad_kernel<<<dim3((cols + 63) / 64, BIAS_SPLIT), 256, 0, st>>>(dA, rows, cols, vec, db);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

static unsigned grid1d(long long n) {
    long long b = (n + 255) / 256;
    const long long cap = 148LL * 32;
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace adock

using namespace adock;

static int gemm_args(GemmArgs& g, int M, int N, int K, const void* A, long long sAm, long long sAk, const void* B,
                     long long sBk, long long sBn, float* C, long long ldc, float beta, const float* bias, int act,
                     float* pre, void* Cb, long long ldcb) {
    ADOCK_CHECK_ARG(M >= 0 && N >= 0 && K >= 0, "negative GEMM size");
    ADOCK_CHECK_ARG(A && B && (C || Cb), "null GEMM operand");
    ADOCK_CHECK_ARG(act == 0 || act == 1, "act must be 0 (none) or 1 (SiLU)");
    ADOCK_CHECK_ARG(!pre || C, "pre-activation output needs C's leading dimension");
    g.M = M; g.N = N; g.K = K;
    g.A = (const __nv_bfloat16*)A; g.sAm = sAm; g.sAk = sAk;
    g.B = (const __nv_bfloat16*)B; g.sBk = sBk; g.sBn = sBn;
    g.C = C; g.ldc = ldc; g.beta = beta; g.bias = bias; g.act = act; g.pre = pre;
    g.Cb = (__nv_bfloat16*)Cb; g.ldcb = ldcb;
    g.dpre = nullptr;
    return ADOCK_OK;
}

static bool aligned(const void* p, size_t n) { return ((uintptr_t)p & (n - 1)) == 0; }

// 16-byte vectors need an aligned base, a vector-multiple stride and extent along the contiguous dimension
static int operand_mode(const void* X, long long s_row, long long s_k, int rows, int K) {
    if (!aligned(X, 16)) return OP_ELEM;
    if (s_k == 1 && s_row % 8 == 0 && K % 8 == 0) return OP_KVEC;
    if (s_row == 1 && s_k % 8 == 0 && rows % 8 == 0) return OP_ROWVEC;
    return OP_ELEM;
}

// Two CTAs of the tcgen05 GEMM fit an SM (shared memory, registers), so their TMEM (at most 2 x 128 of 512 columns)
// always does.
template <int TN>
static int launch_gemm_tc(const GemmArgs& g, int split, cudaStream_t st) {
    const size_t smem = TcSmem<TN>::TOTAL;
    ADOCK_CUDA(cudaFuncSetAttribute(gemm_bf16_tc_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((g.N + TN - 1) / TN, (g.M + TC_BM - 1) / TC_BM, split);
    ADOCK_CHECK_ARG(cfg.gridDim.y < 65536u, "M too large");
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = split;
    cfg.attrs = &attr;
    cfg.numAttrs = split > 1 ? 1 : 0;
    ADOCK_CUDA(cudaLaunchKernelEx(&cfg, gemm_bf16_tc_kernel<TN>, g, operand_mode(g.A, g.sAm, g.sAk, g.M, g.K),
                                  operand_mode(g.B, g.sBn, g.sBk, g.N, g.K)));
    return ADOCK_OK;
}

static int gemm_tc(GemmArgs& g, cudaStream_t st) {
    if (g.M == 0 || g.N == 0) return ADOCK_OK;
    g.vec = (!g.C || (aligned(g.C, 16) && g.ldc % 4 == 0)) && (!g.pre || (aligned(g.pre, 16) && g.ldc % 4 == 0)) &&
            (!g.Cb || (aligned(g.Cb, 8) && g.ldcb % 4 == 0)) && (!g.dpre || (aligned(g.dpre, 16) && g.ldcb % 4 == 0)) &&
            (!g.bias || aligned(g.bias, 16));
    // 128-column tiles read A half as often, 64-column tiles make twice as many CTAs: wide ones once they fill the
    // SMs (forward pass of 8,192 rows, 128 wide tiles or 256 narrow ones: 53.6 or 46.5 us). A cluster splits K where
    // the tiles cover less than half of the SMs and every CTA keeps at least four K steps; the layers' own K (at most
    // five steps) is never split, so their sums keep one order whatever the batch.
    const long long my = (g.M + TC_BM - 1) / TC_BM;
    const bool wide = g.N > 64 && my * ((g.N + 127) / 128) >= sm_count();
    const long long tiles = my * (wide ? (g.N + 127) / 128 : (g.N + 63) / 64);
    const int nk = (g.K + TC_BK - 1) / TC_BK;
    int split = 1;
    while (split < 8 && tiles * split * 2 <= sm_count() && nk >= 8 * split) split *= 2;
    return wide ? launch_gemm_tc<128>(g, split, st) : launch_gemm_tc<64>(g, split, st);
}

extern "C" int adock_gemm_bf16(int M, int N, int K, const void* A, long long sAm, long long sAk, const void* B,
                               long long sBk, long long sBn, float* C, long long ldc, float beta, const float* bias,
                               int act, float* pre, void* Cb, long long ldcb, void* stream) {
    GemmArgs g;
    const int rc = gemm_args(g, M, N, K, A, sAm, sAk, B, sBk, sBn, C, ldc, beta, bias, act, pre, Cb, ldcb);
    if (rc != ADOCK_OK) return rc;
    return gemm_tc(g, (cudaStream_t)stream);
}

extern "C" int adock_gemm_bf16_mma(int M, int N, int K, const void* A, long long sAm, long long sAk, const void* B,
                                   long long sBk, long long sBn, float* C, long long ldc, float beta,
                                   const float* bias, int act, float* pre, void* Cb, long long ldcb, void* stream) {
    GemmArgs g;
    const int rc = gemm_args(g, M, N, K, A, sAm, sAk, B, sBk, sBn, C, ldc, beta, bias, act, pre, Cb, ldcb);
    if (rc != ADOCK_OK) return rc;
    if (M == 0 || N == 0) return ADOCK_OK;
    dim3 grid((N + GN - 1) / GN, (M + GM - 1) / GM);
    ADOCK_CHECK_ARG(grid.y < 65536u, "M too large");
    gemm_bf16_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(g);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

// ------------------------------------------------------------------------------------------------ whole network
namespace adock {
#define NET_IN 320
#define NET_HID 256
#define NET_OUT 64

struct NetBuffers {   // activations and gradients of a batch inside the caller's workspace
    float *pre1, *pre2, *out;
    __nv_bfloat16 *h1, *h2, *dA1, *dA2, *dout;
};

static size_t net_workspace(int B, unsigned char* base, NetBuffers* n) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base ? base + at : nullptr;
        at += (bytes + 255) & ~(size_t)255;
        return p;
    };
    NetBuffers t;
    const size_t b = (size_t)B;
    t.pre1 = (float*)take(b * NET_HID * 4);
    t.pre2 = (float*)take(b * NET_HID * 4);
    t.out = (float*)take(b * NET_OUT * 4);
    t.h1 = (__nv_bfloat16*)take(b * NET_HID * 2);
    t.h2 = (__nv_bfloat16*)take(b * NET_HID * 2);
    t.dA1 = (__nv_bfloat16*)take(b * NET_HID * 2);
    t.dA2 = (__nv_bfloat16*)take(b * NET_HID * 2);
    t.dout = (__nv_bfloat16*)take(b * NET_OUT * 2);
    if (n) *n = t;
    return at;
}

static GemmArgs net_gemm(int M, int N, int K, const void* A, long long sAm, long long sAk, const void* B, long long sBk,
                         long long sBn) {
    GemmArgs g = {};
    g.M = M; g.N = N; g.K = K;
    g.A = (const __nv_bfloat16*)A; g.sAm = sAm; g.sAk = sAk;
    g.B = (const __nv_bfloat16*)B; g.sBk = sBk; g.sBn = sBn;
    return g;
}

// out = (SiLU(SiLU(x W1 + b1) W2 + b2)) W3 + b3; pre1, pre2 may be NULL
static int net_forward(int B, const void* x, const void* const* W, const float* const* b, float* pre1, void* h1, float* pre2,
                       void* h2, float* out, cudaStream_t st) {
    GemmArgs g = net_gemm(B, NET_HID, NET_IN, x, NET_IN, 1, W[0], NET_HID, 1);
    g.bias = b[0]; g.act = 1; g.pre = pre1; g.ldc = NET_HID; g.Cb = (__nv_bfloat16*)h1; g.ldcb = NET_HID;
    int rc = gemm_tc(g, st);
    if (rc) return rc;
    g = net_gemm(B, NET_HID, NET_HID, h1, NET_HID, 1, W[1], NET_HID, 1);
    g.bias = b[1]; g.act = 1; g.pre = pre2; g.ldc = NET_HID; g.Cb = (__nv_bfloat16*)h2; g.ldcb = NET_HID;
    rc = gemm_tc(g, st);
    if (rc) return rc;
    g = net_gemm(B, NET_OUT, NET_HID, h2, NET_HID, 1, W[2], NET_OUT, 1);
    g.bias = b[2]; g.C = out; g.ldc = NET_OUT;
    return gemm_tc(g, st);
}
}  // namespace adock

extern "C" int adock_mlp_forward(int B, const void* x, const void* const* W, const float* const* b, float* pre1, void* h1,
                                 float* pre2, void* h2, float* out, void* stream) {
    ADOCK_CHECK_ARG(B >= 0, "negative batch");
    if (B == 0) return ADOCK_OK;
    ADOCK_CHECK_ARG(x && W && b && W[0] && W[1] && W[2] && b[0] && b[1] && b[2] && h1 && h2 && out, "null argument");
    return net_forward(B, x, W, b, pre1, h1, pre2, h2, out, (cudaStream_t)stream);
}

extern "C" size_t adock_mlp_workspace_bytes(int B) { return net_workspace(B < 0 ? 0 : B, nullptr, nullptr); }

extern "C" int adock_mlp_loss_grad(int B, const void* x, const float* target, const void* const* W, const float* const* b,
                                   int n_comp, void* work, float* const* gW, float* const* gb, float* loss, void* stream) {
    ADOCK_CHECK_ARG(B >= 0, "negative batch");
    ADOCK_CHECK_ARG(n_comp == 1 || n_comp == 3, "n_comp must be 1 or 3 (got %d)", n_comp);
    ADOCK_CHECK_ARG((B == 0 || (x && target && work)) && W && b && gW && gb && loss, "null argument");
    for (int i = 0; i < 3; ++i) ADOCK_CHECK_ARG(W[i] && b[i] && gW[i] && gb[i], "null weight or gradient");
    cudaStream_t st = (cudaStream_t)stream;
    NetBuffers n;
    net_workspace(B, (unsigned char*)work, &n);
    ADOCK_CUDA(cudaMemsetAsync(loss, 0, sizeof(float), st));
    int rc = net_forward(B, x, W, b, n.pre1, n.h1, n.pre2, n.h2, n.out, st);
    if (rc) return rc;
    if (B > 0) launch_nll(n.out, target, B, n_comp, n.dout, loss, st);
    ADOCK_CUDA(cudaGetLastError());
    // per layer: dW = h^T dA, db = column sums of dA, and the layer below's dA = (dA W^T) * SiLU'(pre) in the epilogue
    const void* in[3] = {x, n.h1, n.h2};
    const __nv_bfloat16* dA[3] = {n.dA1, n.dA2, n.dout};
    const int dims[4] = {NET_IN, NET_HID, NET_HID, NET_OUT};
    for (int l = 2; l >= 0; --l) {
        const int ki = dims[l], ko = dims[l + 1];
        GemmArgs g = net_gemm(ki, ko, B, in[l], 1, ki, dA[l], ko, 1);
        g.C = gW[l]; g.ldc = ko;
        rc = gemm_tc(g, st);
        if (rc) return rc;
        rc = launch_bias_grad(dA[l], B, ko, gb[l], st);
        if (rc) return rc;
        if (l == 0) break;
        g = net_gemm(B, ki, ko, dA[l], ko, 1, W[l], 1, ko);
        g.dpre = l == 2 ? n.pre2 : n.pre1;
        g.Cb = (__nv_bfloat16*)dA[l - 1]; g.ldcb = ki;
        rc = gemm_tc(g, st);
        if (rc) return rc;
    }
    return ADOCK_OK;
}

extern "C" int adock_gemm_status(void) {
    int s = 0;
    ADOCK_CUDA(cudaMemcpyFromSymbol(&s, g_tc_status, sizeof(int)));
    if (s != 0) {
        const int zero = 0;
        ADOCK_CUDA(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)));
        set_error("a tcgen05 GEMM gave up waiting for its tensor-core work (mbarrier wait bound)");
        return ADOCK_E_DEVICE;
    }
    return ADOCK_OK;
}

extern "C" int adock_mlp_nll(const float* out, const float* target, int B, int n_comp, void* dout, float* loss,
                             void* stream) {
    ADOCK_CHECK_ARG(out && target && dout && loss && B >= 0, "bad argument");
    ADOCK_CHECK_ARG(n_comp == 1 || n_comp == 3, "n_comp must be 1 or 3 (got %d)", n_comp);
    if (B == 0) return ADOCK_OK;
    launch_nll(out, target, B, n_comp, (__nv_bfloat16*)dout, loss, (cudaStream_t)stream);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

extern "C" int adock_silu_backward(const float* dH, const float* A, long long n, void* dA, void* stream) {
    ADOCK_CHECK_ARG(dH && A && dA && n >= 0, "bad argument");
    if (n == 0) return ADOCK_OK;
    silu_backward_kernel<<<grid1d(n), 256, 0, (cudaStream_t)stream>>>(dH, A, n, (__nv_bfloat16*)dA);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

extern "C" int adock_bias_grad(const void* dA, int rows, int cols, float* db, void* stream) {
    ADOCK_CHECK_ARG(dA && db && rows >= 0 && cols >= 0, "bad argument");
    if (cols == 0) return ADOCK_OK;
    return launch_bias_grad((const __nv_bfloat16*)dA, rows, cols, db, (cudaStream_t)stream);
}

extern "C" int adock_adam(float* p, const float* grad, float* m, float* v, void* pb, long long n, float lr, float b1,
                          float b2, float eps, int step, float wd, void* stream) {
    ADOCK_CHECK_ARG(p && grad && m && v && n >= 0 && step >= 1, "bad argument");
    if (n == 0) return ADOCK_OK;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    adam_kernel<<<grid1d(n), 256, 0, (cudaStream_t)stream>>>(p, grad, m, v, (__nv_bfloat16*)pb, n, lr, b1, b2, eps, c1,
                                                             c2, wd);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

extern "C" int adock_f32_to_bf16(const float* x, void* y, long long n, void* stream) {
    ADOCK_CHECK_ARG(x && y && n >= 0, "bad argument");
    if (n == 0) return ADOCK_OK;
    f32_to_bf16_kernel<<<grid1d(n), 256, 0, (cudaStream_t)stream>>>(x, (__nv_bfloat16*)y, n);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}
