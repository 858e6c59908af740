// mlp.cu -- the learned surrogate: a 3-layer BF16 MLP (n_in -> width ->
// width -> n_out, GELU, FP32 accumulate) trained on the GPU with hand-written
// tensor-core forward/backward kernels and AdamW.
//
// GEMMs run on the 5th-generation tensor cores (tcgen05.mma kind::f16,
// BF16 x BF16 -> FP32 accumulated in tensor memory; k_gemm_tc): every
// product of the forward pass (X W^T), the weight gradients (dZ^T A) and the
// input gradients (dZ W).  Weights are held in FP32 (the
// optimizer's master copy) and in BF16 (the GEMM operand); activations and
// gradients enter the GEMMs as BF16, pre-activations and accumulations stay
// FP32.  This network has no counterpart in the reference: it maps early-time
// spectra of the evolution to late-time magnetic spectra for parameter
// sweeps, and the evolution itself stays the fallback and the reference answer.
//
// Networks whose operands fit shared memory (width a multiple of 16 and at
// most 512, n_in <= 512, n_out <= 128; training batches <= 512), the surrogate's
// among them, run the layer kernels of mlp_layers.cuh; others the general
// GEMM with element-wise kernels.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "ewpt_ctx.cuh"

namespace {

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

struct GemmArgs {
    const __nv_bfloat16* A;
    const __nv_bfloat16* B;
    float* C;
    int M, N, K, lda, ldb, ldc;
    int transA, transB;
    long spin;  // polls before the commit wait gives up, which sets
    int* err;   // (device memory)
};

__device__ __forceinline__ __nv_bfloat16 ldA(const GemmArgs& g, int m, int k) {
    if (m >= g.M || k >= g.K) return __float2bfloat16(0.f);
    return g.transA ? g.A[(int64_t)k * g.lda + m] : g.A[(int64_t)m * g.lda + k];
}
__device__ __forceinline__ __nv_bfloat16 ldB(const GemmArgs& g, int k, int n) {
    if (k >= g.K || n >= g.N) return __float2bfloat16(0.f);
    return g.transB ? g.B[(int64_t)n * g.ldb + k] : g.B[(int64_t)k * g.ldb + n];
}

// ---------------------------------------------------------------- tcgen05
// C[M x N] = op(A) op(B) on the 5th-generation tensor cores: one CTA of 4
// warps per 128 x 64 tile of C, the FP32 accumulator in tensor memory (64
// TMEM columns), K in slabs of 64.  Per slab the 128 threads gather op(A)
// (128 x 64) and op(B)^T (64 x 64) as BF16 into shared memory in the
// canonical K-major layout without swizzle -- 8-row x 16-byte core matrices,
// adjacent along K 128 bytes apart (LBO), 8-row groups 1024 bytes apart
// (SBO) -- (zero outside the matrices, any transposition done by the
// gather), then one thread issues four tcgen05.mma (M 128, N 64, K 16) and
// commits them to an mbarrier that every thread waits on before the slab is
// overwritten.  Finally each warp reads its 32 TMEM lanes (rows) with
// tcgen05.ld and writes C.  Every wait is bounded (g.spin polls, host-set
// by ewpt_mlp_set_wait_limit, default kTcSpin).  A wait that runs out in any
// thread ends the slab loop for the whole CTA (a block-wide vote, so every
// thread leaves the loop at the same barrier), sets the net's flag and skips the
// remaining tensor-core work; before the TMEM columns are freed the CTA waits
// again, with the full kTcSpin limit, for the MMAs already committed.
constexpr int TC_M = 128, TC_N = 64, TC_K = 64;
constexpr long kTcSpin = 1L << 22;

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start, LBO, SBO (bytes), version 1, no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// instruction descriptor, kind::f16: D F32, A and B BF16, both K-major
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, long spin) {
    for (long it = 0; it < spin; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

__global__ void __launch_bounds__(128) k_gemm_tc(GemmArgs g) {
    __shared__ __align__(1024) uint8_t sa[TC_M * TC_K * 2];  // 16 KB
    __shared__ __align__(1024) uint8_t sb[TC_N * TC_K * 2];  // 8 KB
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TC_M, n0 = blockIdx.x * TC_N;
    const uint32_t ubar = tc_smem(&bar);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base)),
                     "r"(TC_N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ubar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    bool ok = true;
    const int nslab = (g.K + TC_K - 1) / TC_K;
    for (int ks = 0; ks < nslab && ok; ++ks) {
        const int k0 = ks * TC_K;
        // gather op(A): row m = tid, 8 chunks of 8 K-elements (one core-matrix row each)
        for (int kc = 0; kc < TC_K / 8; ++kc) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                w[e] = pack_bf16(ldA(g, m0 + tid, k0 + 8 * kc + 2 * e), ldA(g, m0 + tid, k0 + 8 * kc + 2 * e + 1));
            const int off = ((tid >> 3) * (TC_K / 8) + kc) * 128 + (tid & 7) * 16;
            *reinterpret_cast<uint4*>(sa + off) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        // gather op(B)^T: row n, 8 chunks along K; 64 rows x 8 chunks over 128 threads
        for (int q = tid; q < TC_N * (TC_K / 8); q += 128) {
            const int n = q >> 3, kc = q & 7;
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                w[e] = pack_bf16(ldB(g, k0 + 8 * kc + 2 * e, n0 + n), ldB(g, k0 + 8 * kc + 2 * e + 1, n0 + n));
            const int off = ((n >> 3) * (TC_K / 8) + kc) * 128 + (n & 7) * 16;
            *reinterpret_cast<uint4*>(sb + off) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t abase = tc_smem(sa), bbase = tc_smem(sb);
#pragma unroll
            for (int kk = 0; kk < TC_K / 16; ++kk) {
                // K = 16 is two core matrices along K: advance 2 x LBO
                const uint64_t ad = tc_desc(abase + kk * 256, 128, (TC_K / 8) * 128);
                const uint64_t bd = tc_desc(bbase + kk * 256, 128, (TC_K / 8) * 128);
                const uint32_t acc = (ks > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(tc_idesc(TC_M, TC_N)), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ubar)
                         : "memory");
        }
        const bool late = !tc_wait(ubar, ks & 1, g.spin);
        if (__syncthreads_or(late)) {
            // the MMAs of this slab still read shared memory and write TMEM:
            // let them finish before the CTA leaves the loop
            tc_wait(ubar, ks & 1, kTcSpin);
            ok = false;
            if (tid == 0) atomicExch(g.err, 1);
        }
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        const int row = m0 + warp * 32 + lane;
#pragma unroll
        for (int c0 = 0; c0 < TC_N; c0 += 16) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15])
                : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (row < g.M)
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (n0 + c0 + e < g.N) g.C[(int64_t)row * g.ldc + n0 + c0 + e] = __uint_as_float(r[e]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_N) : "memory");
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

}  // namespace

#include "mlp_layers.cuh"

namespace {

// z += bias (in place, z keeps the pre-activation); act = bf16(gelu(z)) or bf16(z)
__global__ void k_bias_act(float* z, const float* __restrict__ bias, __nv_bfloat16* act, int B, int N, int apply) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < (int64_t)B * N;
         q += (int64_t)gridDim.x * blockDim.x) {
        const float v = z[q] + bias[q % N];
        z[q] = v;
        if (act) act[q] = __float2bfloat16(apply ? gelu(v) : v);
    }
}

__global__ void k_to_bf16(const float* __restrict__ x, __nv_bfloat16* y, int64_t n) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        y[q] = __float2bfloat16(x[q]);
}

// dz = 2 (z - y)/(B N) (MSE); per-block partial loss sums
__global__ void k_mse(const float* __restrict__ z, const float* __restrict__ y, float* dzf, __nv_bfloat16* dzb,
                      int64_t n, float scale, float* part) {
    __shared__ float sh[256];
    float s = 0.f;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const float d = z[q] - y[q];
        s += d * d;
        const float g = 2.f * d * scale;
        dzf[q] = g;
        dzb[q] = __float2bfloat16(g);
    }
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// dz = da * gelu'(z)
__global__ void k_gelu_bwd(const float* __restrict__ da, const float* __restrict__ z, float* dzf, __nv_bfloat16* dzb,
                           int64_t n) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const float g = da[q] * gelu_grad(z[q]);
        dzf[q] = g;
        dzb[q] = __float2bfloat16(g);
    }
}

// db[n] = sum_b dz[b][n]
__global__ void k_colsum(const float* __restrict__ dz, float* db, int B, int N) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s = 0.f;
    for (int b = 0; b < B; ++b) s += dz[(int64_t)b * N + n];
    db[n] = s;
}

// No step where a wait of the call's GEMMs ran out (all of them have ended).
__global__ void k_adamw(float* w, const float* __restrict__ g, float* m, float* v, int64_t n, float lr, float b1,
                        float b2, float eps, float wd, float c1, float c2, const int* __restrict__ err) {
    if (*err) return;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const float gq = g[q];
        const float mq = b1 * m[q] + (1.f - b1) * gq;
        const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
        m[q] = mq;
        v[q] = vq;
        w[q] = w[q] - lr * ((mq / c1) / (sqrtf(vq / c2) + eps) + wd * w[q]);
    }
}

__global__ void k_sum_partials(const float* __restrict__ part, int n, float* out) {
    float s = 0.f;
    for (int i = 0; i < n; ++i) s += part[i];
    *out = s;
}

}  // namespace

struct ewpt_mlp {
    int nin = 0, width = 0, nout = 0, maxb = 0, device = 0;
    cudaStream_t st = nullptr;
    int* tc_err = nullptr;      // set by a GEMM whose wait ran out
    int64_t wait_polls = -1;    // limit of the GEMM's tensor-core waits in polls (< 0: default)
    int64_t weight_polls = -1;  // the same in k_weights alone (< 0: wait_polls)
    int64_t np = 0;
    int64_t oW1 = 0, ob1 = 0, oW2 = 0, ob2 = 0, oW3 = 0, ob3 = 0;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    __nv_bfloat16* pb = nullptr;  // bf16 copy of p
    float* xf = nullptr;          // [maxb][nin] input (f32)
    float* yf = nullptr;          // [maxb][nout] target
    __nv_bfloat16* x0 = nullptr;  // [maxb][nin]
    float *z1 = nullptr, *z2 = nullptr, *z3 = nullptr;
    __nv_bfloat16 *a1 = nullptr, *a2 = nullptr;
    float* da = nullptr;          // [maxb][max(width, nout)]
    float* dzf = nullptr;
    __nv_bfloat16* dzb = nullptr;
    float* part = nullptr;        // loss partials
    float* loss = nullptr;
    int64_t t = 0;
    std::string err;
    // layer kernels (mlp_layers.cuh): operand images in one allocation, and
    // mapped page-locked memory for the call's inputs, outputs and status
    bool layers = false;
    int K1 = 0, N3 = 0, Bt = 0;  // n_in and n_out padded, columns of the batch images
    void* images = nullptr;
    __nv_bfloat16 *W1i = nullptr, *W2i = nullptr, *W2t = nullptr, *W3i = nullptr, *W3t = nullptr;
    __nv_bfloat16 *a1i = nullptr, *a2i = nullptr, *dz3i = nullptr, *dz2i = nullptr;
    __nv_bfloat16 *x0T = nullptr, *a1T = nullptr, *a2T = nullptr, *dz1T = nullptr, *dz2T = nullptr, *dz3T = nullptr;
    float *dz1 = nullptr, *dz2 = nullptr, *dz3 = nullptr, *lpart = nullptr;
    int* flag = nullptr;
    int gen = 0;
    int hrows = 0;          // rows of x and z3 in
    float* host = nullptr;  // [0] loss, [1] status, then x, y, z3
    float *hx = nullptr, *hy = nullptr, *hz = nullptr;
    float* mapped = nullptr;  // device address of host
};

namespace {

int mlp_fail(ewpt_mlp* n, int code, const char* msg) {
    if (n) n->err = msg;
    return ewpt_fail(nullptr, code, "%s", msg);
}

int mlp_cuda(ewpt_mlp* n, cudaError_t e, const char* what) {
    if (e == cudaSuccess) {
        // a bounded tensor-core wait that ran out (k_gemm_tc) invalidates the results
        int h = 0;
        if (n && cudaMemcpy(&h, n->tc_err, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess && h) {
            cudaMemsetAsync(n->tc_err, 0, sizeof h, n->st);
            return mlp_fail(n, EWPT_ERR_TIMEOUT, "a tensor-core wait in the MLP GEMM ran out (results invalid)");
        }
        return EWPT_OK;
    }
    std::string s = std::string(what) + ": " + cudaGetErrorString(e);
    return mlp_fail(n, e == cudaErrorMemoryAllocation ? EWPT_ERR_OOM : EWPT_ERR_CUDA, s.c_str());
}

cudaError_t gemm(const ewpt_mlp* n, const __nv_bfloat16* A, int lda, int transA, const __nv_bfloat16* B, int ldb,
                 int transB, float* C, int ldc, int M, int N, int K) {
    const cudaStream_t st = n->st;
    GemmArgs g{A, B, C, M, N, K, lda, ldb, ldc, transA, transB, n->wait_polls < 0 ? kTcSpin : (long)n->wait_polls, n->tc_err};
    const dim3 gr((N + TC_N - 1) / TC_N, (M + TC_M - 1) / TC_M);
    k_gemm_tc<<<gr, 128, 0, st>>>(g);
    return cudaGetLastError();
}

const int kEW = 1216;  // elementwise grid

cudaError_t refresh_bf16(ewpt_mlp* n) {
    k_to_bf16<<<kEW, 256, 0, n->st>>>(n->p, n->pb, n->np);
    return cudaGetLastError();
}

// Forward pass on the batch already in n->xf; leaves z1, z2, z3, a1, a2.
cudaError_t forward(ewpt_mlp* n, int B) {
    cudaError_t e;
    k_to_bf16<<<kEW, 256, 0, n->st>>>(n->xf, n->x0, (int64_t)B * n->nin);
    e = gemm(n, n->x0, n->nin, 0, n->pb + n->oW1, n->nin, 1, n->z1, n->width, B, n->width, n->nin);
    if (e) return e;
    k_bias_act<<<kEW, 256, 0, n->st>>>(n->z1, n->p + n->ob1, n->a1, B, n->width, 1);
    e = gemm(n, n->a1, n->width, 0, n->pb + n->oW2, n->width, 1, n->z2, n->width, B, n->width, n->width);
    if (e) return e;
    k_bias_act<<<kEW, 256, 0, n->st>>>(n->z2, n->p + n->ob2, n->a2, B, n->width, 1);
    e = gemm(n, n->a2, n->width, 0, n->pb + n->oW3, n->width, 1, n->z3, n->nout, B, n->nout, n->width);
    if (e) return e;
    k_bias_act<<<kEW, 256, 0, n->st>>>(n->z3, n->p + n->ob3, nullptr, B, n->nout, 0);
    return cudaGetLastError();
}

// Loss and gradients into n->g (target batch in n->yf).
cudaError_t backward(ewpt_mlp* n, int B) {
    cudaError_t e;
    const int W = n->width, O = n->nout, I = n->nin;
    const int nb = 64;
    k_mse<<<nb, 256, 0, n->st>>>(n->z3, n->yf, n->dzf, n->dzb, (int64_t)B * O, 1.f / ((float)B * O), n->part);
    k_sum_partials<<<1, 1, 0, n->st>>>(n->part, nb, n->loss);
    // layer 3
    e = gemm(n, n->dzb, O, 1, n->a2, W, 0, n->g + n->oW3, W, O, W, B);  // dW3 = dZ3^T A2
    if (e) return e;
    k_colsum<<<(O + 127) / 128, 128, 0, n->st>>>(n->dzf, n->g + n->ob3, B, O);
    e = gemm(n, n->dzb, O, 0, n->pb + n->oW3, W, 0, n->da, W, B, W, O);  // dA2 = dZ3 W3
    if (e) return e;
    k_gelu_bwd<<<kEW, 256, 0, n->st>>>(n->da, n->z2, n->dzf, n->dzb, (int64_t)B * W);
    // layer 2
    e = gemm(n, n->dzb, W, 1, n->a1, W, 0, n->g + n->oW2, W, W, W, B);  // dW2 = dZ2^T A1
    if (e) return e;
    k_colsum<<<(W + 127) / 128, 128, 0, n->st>>>(n->dzf, n->g + n->ob2, B, W);
    e = gemm(n, n->dzb, W, 0, n->pb + n->oW2, W, 0, n->da, W, B, W, W);  // dA1 = dZ2 W2
    if (e) return e;
    k_gelu_bwd<<<kEW, 256, 0, n->st>>>(n->da, n->z1, n->dzf, n->dzb, (int64_t)B * W);
    // layer 1
    e = gemm(n, n->dzb, W, 1, n->x0, I, 0, n->g + n->oW1, I, W, I, B);  // dW1 = dZ1^T X0
    if (e) return e;
    k_colsum<<<(W + 127) / 128, 128, 0, n->st>>>(n->dzf, n->g + n->ob1, B, W);
    return cudaGetLastError();
}

// ---- layer kernels
constexpr int kMappedHead = 32;  // floats before x in the mapped buffer
// Layer 1 reads a batch's inputs once for each of its width / 16 column tiles:
// from the mapped buffer while that is at most so many floats, else from a copy
// in device memory.  Forward pass, us, mapped / copied: 84-256-40 128 rows 41 / 42,
// 256 rows 46 / 48, 512 rows 67 / 51, 8192 rows 567 / 183; 512-512-128 32 rows 53 / 54,
// 128 rows 89 / 66, 8192 rows 4146 / 748 (element-wise kernels and general GEMM: 299
// and 899 at 8192).
constexpr int64_t kHostReads = 3 << 17;

bool layers_fit(const ewpt_mlp* n) {
    return n->width % LN == 0 && n->width <= kLayerMaxK && n->nin <= kLayerMaxK && n->nout <= LM;
}

cudaError_t layers_alloc(ewpt_mlp* n) {
    const int W = n->width;
    n->K1 = round_up(n->nin, 16);
    n->N3 = round_up(n->nout, LN);
    n->Bt = round_up(std::min(n->maxb, kLayerMaxK), 16);
    const int64_t Mp = round_up(n->maxb, LM), Wm = round_up(W, LM);
    // bf16 images, then the FP32 arrays and the flag; every piece a multiple of 128 bytes
    struct Piece {
        void** p;
        int64_t bytes;
    } pieces[] = {{(void**)&n->W1i, (int64_t)W * n->K1 * 2},
                  {(void**)&n->W2i, (int64_t)W * W * 2},
                  {(void**)&n->W2t, (int64_t)W * W * 2},
                  {(void**)&n->W3i, (int64_t)n->N3 * W * 2},
                  {(void**)&n->W3t, (int64_t)W * n->N3 * 2},
                  {(void**)&n->a1i, Mp * W * 2},
                  {(void**)&n->a2i, Mp * W * 2},
                  {(void**)&n->dz3i, Mp * n->N3 * 2},
                  {(void**)&n->dz2i, Mp * W * 2},
                  {(void**)&n->x0T, (int64_t)round_up(n->nin, LN) * n->Bt * 2},
                  {(void**)&n->a1T, (int64_t)W * n->Bt * 2},
                  {(void**)&n->a2T, (int64_t)W * n->Bt * 2},
                  {(void**)&n->dz1T, Wm * n->Bt * 2},
                  {(void**)&n->dz2T, Wm * n->Bt * 2},
                  {(void**)&n->dz3T, (int64_t)LM * n->Bt * 2},
                  {(void**)&n->dz1, (int64_t)n->maxb * W * 4},
                  {(void**)&n->dz2, (int64_t)n->maxb * W * 4},
                  {(void**)&n->dz3, (int64_t)n->maxb * n->nout * 4},
                  {(void**)&n->lpart, Mp / LM * (n->N3 / LN) * (LT / 32) * 4},
                  {(void**)&n->flag, 4}};
    int64_t total = 0;
    for (const Piece& q : pieces) total += (q.bytes + 127) / 128 * 128;
    cudaError_t e = cudaMalloc(&n->images, total);
    if (e == cudaSuccess) e = cudaMemsetAsync(n->images, 0, total, n->st);  // the padding stays zero
    int64_t off = 0;
    for (const Piece& q : pieces) {
        *q.p = static_cast<char*>(n->images) + off;
        off += (q.bytes + 127) / 128 * 128;
    }
    n->hrows = (int)std::min<int64_t>(std::max<int64_t>(kHostReads / ((int64_t)n->nin * (W / LN)), 1), n->maxb);
    const int64_t targets = (int64_t)std::min(n->maxb, kLayerMaxK) * n->nout;
    if (e == cudaSuccess)
        e = cudaHostAlloc((void**)&n->host, (kMappedHead + targets + (int64_t)n->hrows * (n->nin + n->nout)) * 4,
                          cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&n->mapped, n->host, 0);
    n->hx = n->host + kMappedHead;
    n->hy = n->hx + (int64_t)n->hrows * n->nin;
    n->hz = n->hy + targets;
    const int smem = (LM + LN) * kLayerMaxK * 2;
    const void* kernels[] = {(const void*)k_layer<kForward>, (const void*)k_layer<kOutput>,
                             (const void*)k_layer<kBackward>, (const void*)k_weights};
    for (const void* k : kernels)
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

// set_params: the weight images
cudaError_t layers_pack(ewpt_mlp* n) {
    const int W = n->width;
    k_pack<<<152, 256, 0, n->st>>>(n->p + n->oW1, W, n->nin, n->W1i, n->K1, nullptr, 0);
    k_pack<<<152, 256, 0, n->st>>>(n->p + n->oW2, W, W, n->W2i, W, n->W2t, W);
    k_pack<<<152, 256, 0, n->st>>>(n->p + n->oW3, n->nout, W, n->W3i, W, n->W3t, n->N3);
    return cudaGetLastError();
}

// dependent: the kernel may start before the previous one of the stream ends
template <class Args>
cudaError_t launch(const ewpt_mlp* n, void (*k)(Args), dim3 grid, int smem, const Args& a, bool dependent) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(LT);
    c.dynamicSmemBytes = smem;
    c.stream = n->st;
    c.attrs = &at;
    c.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&c, k, a);
}

// The layers on the inputs x and the targets in the mapped buffer; train: loss
// and weight gradients into n->g, and (adam) one AdamW step.
cudaError_t layers_run(ewpt_mlp* n, const float* x, int B, bool train, bool adam, float lr, float wd, float c1,
                       float c2) {
    cudaError_t e = cudaSuccess;
    if (B <= n->hrows)
        std::memcpy(n->hx, x, (size_t)B * n->nin * 4);
    else
        e = cudaMemcpyAsync(n->xf, x, (size_t)B * n->nin * 4, cudaMemcpyHostToDevice, n->st);
    if (e != cudaSuccess) return e;
    const int W = n->width, I = n->nin, O = n->nout, Bp = round_up(B, 16);
    const unsigned my = (unsigned)((B + LM - 1) / LM);
    n->host[0] = 0.f;
    reinterpret_cast<int*>(n->host)[1] = 0;
    ++n->gen;
    const Status st{reinterpret_cast<volatile int*>(n->mapped) + 1, n->flag, n->gen,
                    n->wait_polls < 0 ? kTcSpin : (long)n->wait_polls};
    LayerArgs b{};
    b.batch = B;
    b.nin = I;
    b.Bp = Bp;
    b.train = train;
    b.st = st;
    LayerArgs f1 = b, f2 = b, f3 = b, b2 = b, b1 = b;
    f1.x = B <= n->hrows ? n->mapped + kMappedHead : n->xf;
    f1.W = n->W1i, f1.bias = n->p + n->ob1, f1.N = W, f1.Kp = n->K1, f1.z = n->z1, f1.out = n->a1i, f1.outK = W;
    f2.A = n->a1i, f2.W = n->W2i, f2.bias = n->p + n->ob2, f2.N = W, f2.Kp = W, f2.z = n->z2, f2.out = n->a2i, f2.outK = W;
    f3.A = n->a2i, f3.W = n->W3i, f3.bias = n->p + n->ob3, f3.N = O, f3.Kp = W, f3.zo = n->z3;
    if (train) {
        f1.xT = n->x0T, f1.outT = n->a1T, f2.outT = n->a2T;
        f3.y = n->mapped + (n->hy - n->host), f3.scale = 1.f / ((float)B * O), f3.loss = n->lpart, f3.dz = n->dz3;
        f3.out = n->dz3i, f3.outK = n->N3, f3.outT = n->dz3T;
    }
    auto smem = [](int K) { return (LM + LN) * K * 2; };
    e = launch(n, k_layer<kForward>, dim3(W / LN, my), smem(f1.Kp), f1, false);
    if (e == cudaSuccess) e = launch(n, k_layer<kForward>, dim3(W / LN, my), smem(W), f2, true);
    if (e == cudaSuccess) e = launch(n, k_layer<kOutput>, dim3(n->N3 / LN, my), smem(W), f3, true);
    if (!train || e != cudaSuccess) return e;
    b2.A = n->dz3i, b2.W = n->W3t, b2.N = W, b2.Kp = n->N3, b2.z = n->z2, b2.dz = n->dz2, b2.out = n->dz2i, b2.outK = W;
    b2.outT = n->dz2T;
    b1.A = n->dz2i, b1.W = n->W2t, b1.N = W, b1.Kp = W, b1.z = n->z1, b1.dz = n->dz1, b1.outT = n->dz1T;
    e = launch(n, k_layer<kBackward>, dim3(W / LN, my), smem(n->N3), b2, true);
    if (e == cudaSuccess) e = launch(n, k_layer<kBackward>, dim3(W / LN, my), smem(W), b1, true);
    WeightArgs w{};
    const int tw = round_up(W, LM) / LM, n1 = round_up(I, LN) / LN, nW = W / LN;
    w.w[0] = WeightGrad{n->dz2T, n->a1T, n->dz2, W, W, nW, 0, n->oW2, n->ob2};
    w.w[1] = WeightGrad{n->dz1T, n->x0T, n->dz1, W, I, n1, tw * nW, n->oW1, n->ob1};
    w.w[2] = WeightGrad{n->dz3T, n->a2T, n->dz3, O, W, nW, tw * (nW + n1), n->oW3, n->ob3};
    w.batch = B, w.Bp = Bp, w.nloss = (int)my * (n->N3 / LN) * (LT / 32), w.loss_part = n->lpart;
    w.loss = n->mapped;
    w.g = n->g;
    w.st = st;
    if (n->weight_polls >= 0) w.st.spin = (long)n->weight_polls;
    if (e == cudaSuccess)
        e = launch(n, k_weights, dim3(tw * (nW + n1) + nW), std::max(smem(Bp), LM * (LN + 1) * 4), w, true);
    if (!adam || e != cudaSuccess) return e;
    StepArgs s{};
    s.w[0] = StepWeights{n->oW1, W, I, n->W1i, nullptr, n->K1, 0};
    s.w[1] = StepWeights{n->oW2, W, W, n->W2i, n->W2t, W, W};
    s.w[2] = StepWeights{n->oW3, O, W, n->W3i, n->W3t, W, n->N3};
    s.np = n->np, s.g = n->g, s.p = n->p, s.m = n->m, s.v = n->v, s.pb = n->pb;
    s.lr = lr, s.b1 = 0.9f, s.b2 = 0.999f, s.eps = 1e-8f, s.wd = wd, s.c1 = c1, s.c2 = c2;
    s.st = st;
    return launch(n, k_step, dim3((unsigned)std::min<int64_t>((n->np + LT - 1) / LT, 1216)), 0, s, true);
}

// after the stream has been waited for
int layers_done(ewpt_mlp* n, cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        std::string s = std::string(what) + ": " + cudaGetErrorString(e);
        return mlp_fail(n, e == cudaErrorMemoryAllocation ? EWPT_ERR_OOM : EWPT_ERR_CUDA, s.c_str());
    }
    if (reinterpret_cast<volatile int*>(n->host)[1])
        return mlp_fail(n, EWPT_ERR_TIMEOUT, "a tensor-core wait in the MLP layers ran out (results invalid)");
    return EWPT_OK;
}

int check_batch(ewpt_mlp* n, int B) {
    if (!n) return ewpt_fail(nullptr, EWPT_ERR_ARG, "mlp is NULL");
    if (B < 1 || B > n->maxb) return mlp_fail(n, EWPT_ERR_ARG, "batch size out of range (1..max_batch)");
    cudaSetDevice(n->device);
    return EWPT_OK;
}

cudaError_t upload(ewpt_mlp* n, float* dst, const float* src, int64_t count) {
    return cudaMemcpyAsync(dst, src, count * 4, cudaMemcpyHostToDevice, n->st);
}

}  // namespace

extern "C" {

int ewpt_mlp_create(int32_t n_in, int32_t width, int32_t n_out, int32_t max_batch, int32_t device, ewpt_mlp** out) {
    if (!out) return ewpt_fail(nullptr, EWPT_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (n_in < 1 || width < 1 || n_out < 1 || max_batch < 1 || n_in > 65536 || width > 65536 || n_out > 65536)
        return ewpt_fail(nullptr, EWPT_ERR_ARG, "bad MLP dimensions");
    ewpt_mlp* n = new ewpt_mlp();
    n->nin = n_in;
    n->width = width;
    n->nout = n_out;
    n->maxb = max_batch;
    n->device = device;
    n->oW1 = 0;
    n->ob1 = n->oW1 + (int64_t)width * n_in;
    n->oW2 = n->ob1 + width;
    n->ob2 = n->oW2 + (int64_t)width * width;
    n->oW3 = n->ob2 + width;
    n->ob3 = n->oW3 + (int64_t)n_out * width;
    n->np = n->ob3 + n_out;
    const int64_t wa = std::max(width, n_out);
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&n->st, cudaStreamNonBlocking);
    auto A = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
        if (e == cudaSuccess) e = cudaMemsetAsync(*p, 0, bytes, n->st);
    };
    A((void**)&n->p, n->np * 4);
    A((void**)&n->g, n->np * 4);
    A((void**)&n->m, n->np * 4);
    A((void**)&n->v, n->np * 4);
    A((void**)&n->pb, n->np * 2);
    A((void**)&n->xf, (size_t)max_batch * n_in * 4);
    A((void**)&n->yf, (size_t)max_batch * n_out * 4);
    A((void**)&n->x0, (size_t)max_batch * n_in * 2);
    A((void**)&n->z1, (size_t)max_batch * width * 4);
    A((void**)&n->z2, (size_t)max_batch * width * 4);
    A((void**)&n->z3, (size_t)max_batch * n_out * 4);
    A((void**)&n->a1, (size_t)max_batch * width * 2);
    A((void**)&n->a2, (size_t)max_batch * width * 2);
    A((void**)&n->da, (size_t)max_batch * wa * 4);
    A((void**)&n->dzf, (size_t)max_batch * wa * 4);
    A((void**)&n->dzb, (size_t)max_batch * wa * 2);
    A((void**)&n->part, 64 * 4);
    A((void**)&n->loss, 4);
    A((void**)&n->tc_err, 4);
    n->layers = layers_fit(n);
    if (e == cudaSuccess && n->layers) e = layers_alloc(n);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
    int rc = mlp_cuda(nullptr, e, "mlp allocation");
    if (rc) {
        ewpt_mlp_destroy(n);
        return rc;
    }
    *out = n;
    return EWPT_OK;
}

int ewpt_mlp_destroy(ewpt_mlp* n) {
    if (!n) return EWPT_OK;
    cudaSetDevice(n->device);
    if (n->st) cudaStreamSynchronize(n->st);
    void* bufs[] = {n->p, n->g, n->m, n->v, n->pb, n->xf, n->yf, n->x0, n->z1, n->z2, n->z3,
                    n->a1, n->a2, n->da, n->dzf, n->dzb, n->part, n->loss, n->tc_err};
    for (void* b : bufs) cudaFree(b);
    cudaFree(n->images);
    cudaFreeHost(n->host);
    if (n->st) cudaStreamDestroy(n->st);
    delete n;
    return EWPT_OK;
}

const char* ewpt_mlp_last_error(const ewpt_mlp* n) { return n ? n->err.c_str() : ewpt_last_error(nullptr); }

int64_t ewpt_mlp_num_params(const ewpt_mlp* n) { return n ? n->np : -1; }

int ewpt_mlp_set_wait_limit(ewpt_mlp* n, int64_t polls) {
    if (!n) return ewpt_fail(nullptr, EWPT_ERR_ARG, "net is NULL");
    n->wait_polls = polls < 0 ? -1 : polls;
    return EWPT_OK;
}

int ewpt_mlp_set_weight_wait_limit(ewpt_mlp* n, int64_t polls) {
    if (!n) return ewpt_fail(nullptr, EWPT_ERR_ARG, "net is NULL");
    n->weight_polls = polls < 0 ? -1 : polls;
    return EWPT_OK;
}

int ewpt_mlp_set_params(ewpt_mlp* n, const float* params) {
    if (!n || !params) return ewpt_fail(nullptr, EWPT_ERR_ARG, "NULL argument");
    for (int64_t q = 0; q < n->np; ++q)
        if (!std::isfinite(params[q])) return mlp_fail(n, EWPT_ERR_ARG, "non-finite parameter");
    cudaSetDevice(n->device);
    cudaError_t e = cudaMemcpyAsync(n->p, params, n->np * 4, cudaMemcpyHostToDevice, n->st);
    if (e == cudaSuccess) e = cudaMemsetAsync(n->m, 0, n->np * 4, n->st);
    if (e == cudaSuccess) e = cudaMemsetAsync(n->v, 0, n->np * 4, n->st);
    if (e == cudaSuccess) e = refresh_bf16(n);
    if (e == cudaSuccess && n->layers) e = layers_pack(n);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
    n->t = 0;
    return mlp_cuda(n, e, "mlp set_params");
}

int ewpt_mlp_get_params(ewpt_mlp* n, float* params) {
    if (!n || !params) return ewpt_fail(nullptr, EWPT_ERR_ARG, "NULL argument");
    cudaSetDevice(n->device);
    cudaError_t e = cudaMemcpyAsync(params, n->p, n->np * 4, cudaMemcpyDeviceToHost, n->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
    return mlp_cuda(n, e, "mlp get_params");
}

int ewpt_mlp_forward(ewpt_mlp* n, const float* x, int32_t batch, float* y) {
    int rc = check_batch(n, batch);
    if (rc) return rc;
    if (!x || !y) return mlp_fail(n, EWPT_ERR_ARG, "NULL argument");
    if (n->layers) {
        const size_t out = (size_t)batch * n->nout * 4;
        const bool staged = batch <= n->hrows;
        cudaError_t e = layers_run(n, x, batch, false, false, 0.f, 0.f, 1.f, 1.f);
        if (e == cudaSuccess) e = cudaMemcpyAsync(staged ? n->hz : y, n->z3, out, cudaMemcpyDeviceToHost, n->st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
        rc = layers_done(n, e, "mlp forward");
        if (!rc && staged) std::memcpy(y, n->hz, out);
        return rc;
    }
    cudaError_t e = upload(n, n->xf, x, (int64_t)batch * n->nin);
    if (e == cudaSuccess) e = forward(n, batch);
    if (e == cudaSuccess) e = cudaMemcpyAsync(y, n->z3, (size_t)batch * n->nout * 4, cudaMemcpyDeviceToHost, n->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
    return mlp_cuda(n, e, "mlp forward");
}

int ewpt_mlp_gradients(ewpt_mlp* n, const float* x, const float* y, int32_t batch, float* grads, float* loss) {
    int rc = check_batch(n, batch);
    if (rc) return rc;
    if (!x || !y || !grads) return mlp_fail(n, EWPT_ERR_ARG, "NULL argument");
    if (n->layers && batch <= kLayerMaxK) {
        std::memcpy(n->hy, y, (size_t)batch * n->nout * 4);
        cudaError_t e = layers_run(n, x, batch, true, false, 0.f, 0.f, 1.f, 1.f);
        if (e == cudaSuccess) e = cudaMemcpyAsync(grads, n->g, n->np * 4, cudaMemcpyDeviceToHost, n->st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
        if (loss) *loss = n->host[0] / ((float)batch * n->nout);
        return layers_done(n, e, "mlp gradients");
    }
    cudaError_t e = upload(n, n->xf, x, (int64_t)batch * n->nin);
    if (e == cudaSuccess) e = upload(n, n->yf, y, (int64_t)batch * n->nout);
    if (e == cudaSuccess) e = forward(n, batch);
    if (e == cudaSuccess) e = backward(n, batch);
    if (e == cudaSuccess) e = cudaMemcpyAsync(grads, n->g, n->np * 4, cudaMemcpyDeviceToHost, n->st);
    float l = 0.f;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&l, n->loss, 4, cudaMemcpyDeviceToHost, n->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
    if (loss) *loss = l / ((float)batch * n->nout);
    return mlp_cuda(n, e, "mlp gradients");
}

int ewpt_mlp_train_step(ewpt_mlp* n, const float* x, const float* y, int32_t batch, float lr, float weight_decay,
                        float* loss) {
    int rc = check_batch(n, batch);
    if (rc) return rc;
    if (!x || !y) return mlp_fail(n, EWPT_ERR_ARG, "NULL argument");
    if (!std::isfinite(lr) || !std::isfinite(weight_decay)) return mlp_fail(n, EWPT_ERR_ARG, "non-finite lr/wd");
    if (n->layers && batch <= kLayerMaxK) {
        std::memcpy(n->hy, y, (size_t)batch * n->nout * 4);
        const int64_t t = n->t + 1;
        cudaError_t e = layers_run(n, x, batch, true, true, lr, weight_decay, 1.f - std::pow(0.9f, (float)t),
                                   1.f - std::pow(0.999f, (float)t));
        if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
        if (loss) *loss = n->host[0] / ((float)batch * n->nout);
        rc = layers_done(n, e, "mlp train_step");
        if (!rc) n->t = t;
        return rc;
    }
    cudaError_t e = upload(n, n->xf, x, (int64_t)batch * n->nin);
    if (e == cudaSuccess) e = upload(n, n->yf, y, (int64_t)batch * n->nout);
    if (e == cudaSuccess) e = forward(n, batch);
    if (e == cudaSuccess) e = backward(n, batch);
    const int64_t t = n->t + 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)t), c2 = 1.f - std::pow(b2, (float)t);
    if (e == cudaSuccess) {
        k_adamw<<<kEW, 256, 0, n->st>>>(n->p, n->g, n->m, n->v, n->np, lr, b1, b2, 1e-8f, weight_decay, c1, c2, n->tc_err);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = refresh_bf16(n);
    if (e == cudaSuccess && n->layers) e = layers_pack(n);
    float l = 0.f;
    if (e == cudaSuccess && loss) e = cudaMemcpyAsync(&l, n->loss, 4, cudaMemcpyDeviceToHost, n->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(n->st);
    if (loss) *loss = l / ((float)batch * n->nout);
    rc = mlp_cuda(n, e, "mlp train_step");
    if (!rc) n->t = t;
    return rc;
}

}  // extern "C"
