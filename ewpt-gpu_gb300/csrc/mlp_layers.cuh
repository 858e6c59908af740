// mlp_layers.cuh -- the surrogate network's layers with their element-wise
// work in the GEMM epilogues, for networks whose operands fit shared memory.
//
// A training step at the surrogate's size (84-256-256-40, batches of 128) is
// bound by latency: 0.06 GFLOP, 1 MB.  As 11 general GEMMs (k_gemm_tc, 25 us
// each, most of it the scalar gather of the operands) and 13 element-wise
// launches it took 267 us, and takes 55 now (forward pass 137 and 41).  Here it is
// seven launches:
//   layer 1, layer 2    Z = A W^T + b, A' = gelu(Z)
//   layer 3             Z3, the loss and dZ3
//   back 2, back 1      dZ = (dZ' W) gelu'(Z)
//   weights             all three dW = dZ^T A with the bias sums
//   AdamW               unless a wait of the call ran out
// Every operand lies in global memory as the tensor cores read it (K-major
// core matrices of 8 rows x 16 bytes, no swizzle), written by the kernel that
// makes it: an epilogue stores the activations once with K along the features,
// for the next layer, and once with K along the batch, for the weight
// gradients, and AdamW stores the weights in both orders.  So a CTA's operands
// are two bulk copies, and one thread issues the MMAs of the whole K.  Weight
// tiles are fetched before the wait for the previous kernel (programmatic
// dependent launch).
//
// The accumulation order along K is k_gemm_tc's (K = 16 per MMA, in order).
//
// Waits are bounded as in k_gemm_tc: one that runs out ends the CTA's work
// after its copies and MMAs in flight have landed, and marks the call.  The
// parameters are stepped by a kernel of their own, which reads the mark after the
// last of the waits: a step is taken whole or not at all.
#pragma once
#include <cuda_bf16.h>

namespace {

// Tile of an output: 128 x 16, by 256 threads (a warp reads 32 rows x 8
// columns of the accumulator).  Narrow tiles cost little, since the operands
// come from L2, and keep the element-wise work of a thread short: with 128 x
// 32 by 128 threads the layers took 12-18 us and the weights 28 us each.
constexpr int LM = 128, LN = 16, LT = 256;
constexpr int kTmemCols = 32;     // the smallest allocation
constexpr int kLayerMaxK = 512;   // (128 + 16) rows x 512 x 2 B = 144 KB of shared memory

__host__ __device__ constexpr int round_up(int v, int m) { return (v + m - 1) / m * m; }

// element (r, k) of an operand image with Kp (a multiple of 16) columns
__host__ __device__ __forceinline__ int64_t img(int r, int k, int Kp) {
    return ((int64_t)(r >> 3) * (Kp >> 3) + (k >> 3)) * 64 + (r & 7) * 8 + (k & 7);
}

struct Status {
    volatile int* host;  // mapped: nonzero = a wait of this call ran out
    int* dev;            // = gen of the last call that had one
    int gen;
    long spin;
};

__device__ __forceinline__ void mark(const Status& s) {
    *s.dev = s.gen;
    *s.host = 1;
    __threadfence_system();
}

// Shared state of a tile: barriers, tensor memory, operand tiles.
struct Tile {
    uint64_t ld, mma;
    uint32_t tmem;
};

__device__ __forceinline__ void tile_begin(Tile& t) {
    const int warp = threadIdx.x >> 5;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&t.tmem)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&t.ld)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&t.mma)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tile_expect(Tile& t, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&t.ld)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tile_copy(Tile& t, void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     tc_smem(dst)),
                 "l"(src), "r"(bytes), "r"(tc_smem(&t.ld))
                 : "memory");
}
// Every thread; false (for the whole CTA) once the wait has run out and what
// it waited for has landed.
__device__ __forceinline__ bool tile_wait(uint64_t& bar, const Status& st) {
    const bool late = !tc_wait(tc_smem(&bar), 0, st.spin);
    if (!__syncthreads_or(late)) return true;
    tc_wait(tc_smem(&bar), 0, kTcSpin);
    if (threadIdx.x == 0) mark(st);
    return false;
}

// D[128 x 16] = A[128 x Kp] B[16 x Kp]^T on the operand tiles in shared memory
__device__ __forceinline__ bool tile_mma(Tile& t, const void* A, const void* B, int Kp, const Status& st) {
    if (threadIdx.x == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = tc_smem(A), b = tc_smem(B), sbo = (uint32_t)Kp * 16;
        for (int kk = 0; kk < Kp / 16; ++kk) {
            const uint64_t ad = tc_desc(a + kk * 256, 128, sbo), bd = tc_desc(b + kk * 256, 128, sbo);
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(t.tmem),
                "l"(ad), "l"(bd), "r"(tc_idesc(LM, LN)), "r"(kk > 0 ? 1u : 0u)
                : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         tc_smem(&t.mma))
                     : "memory");
    }
    const bool ok = tile_wait(t.mma, st);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ok;
}

// This thread's 8 values of the accumulator: row tile_row(), columns from
// tile_col() on (a warp reads the 32 lanes of its number modulo 4)
__device__ __forceinline__ int tile_row() { return threadIdx.x & 127; }
__device__ __forceinline__ int tile_col() { return (threadIdx.x >> 7) * 8; }
__device__ __forceinline__ void tile_read(const Tile& t, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(t.tmem + ((uint32_t)(tile_row() & ~31) << 16) + (uint32_t)tile_col()));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[e]);
}

__device__ __forceinline__ void tile_end(const Tile& t) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((threadIdx.x >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(t.tmem), "r"(kTmemCols) : "memory");
}

__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

struct LayerArgs {
    const __nv_bfloat16* A;  // operand image [rows][Kp], or null: x
    const float* x;          // FP32 rows of nin (layer 1)
    const __nv_bfloat16* W;  // weight image [N][Kp]
    const float* bias;
    int batch, nin, N, Kp;   // N: features, of which n0 .. n0 + 15 here
    int Bp;                  // columns of the images with K along the batch
    int train;
    float* z;                // [batch][N] (read by the backward layers)
    float* zo;               // layer 3: the output
    const float* y;          // layer 3, training: targets [batch][N]
    float scale;             // 1 / (batch N)
    float* loss;             // per-warp sums of squares
    float* dz;               // [batch][N] FP32 gradients of the pre-activations
    __nv_bfloat16* out;      // image [rows][outK] of what the next layer reads, or null
    int outK;
    __nv_bfloat16* outT;     // image [N][Bp] for the weight gradients, or null
    __nv_bfloat16* xT;       // layer 1: image [nin][Bp] of x, or null
    Status st;
};

enum LayerKind { kForward, kOutput, kBackward };

template <LayerKind KIND>
__global__ void __launch_bounds__(LT) k_layer(const __grid_constant__ LayerArgs g) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ Tile t;
    uint8_t *sa = smem, *sb = smem + LM * g.Kp * 2;
    const int tid = threadIdx.x, m0 = blockIdx.y * LM, n0 = blockIdx.x * LN;
    tile_begin(t);
    // not before this CTA holds its tensor memory: the next kernel's CTAs wait
    // for this kernel with theirs in hand
    dep_launch();
    const uint32_t ba = LM * g.Kp * 2, bb = LN * g.Kp * 2;
    if (tid == 0) {
        tile_expect(t, bb + (g.A ? ba : 0));
        tile_copy(t, sb, g.W + img(n0, 0, g.Kp), bb);  // weights: no earlier kernel of the call writes them
    }
    dep_wait();
    if (g.A) {
        if (tid == 0) tile_copy(t, sa, g.A + img(m0, 0, g.Kp), ba);
    } else {
        const int nc = g.Kp / 8;
        const float* __restrict__ x = g.x;  // the caller's rows, in host memory
#pragma unroll 3
        for (int q = tid; q < LM * nc; q += LT) {
            const int r = q / nc, k0 = (q - r * nc) * 8, row = m0 + r;
            __nv_bfloat16 v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                v[e] = __float2bfloat16(row < g.batch && k0 + e < g.nin ? __ldg(x + (int64_t)row * g.nin + k0 + e) : 0.f);
            *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(sa) + img(r, k0, g.Kp)) =
                *reinterpret_cast<const uint4*>(v);
            if (g.xT && (k0 >> 3) % gridDim.x == blockIdx.x && row < g.Bp)
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (k0 + e < g.nin) g.xT[img(k0 + e, row, g.Bp)] = v[e];
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    // what the epilogue reads of its elements, on its way while the tiles and
    // the MMAs are (the targets come from host memory)
    const int row = m0 + tile_row(), n1 = n0 + tile_col();
    const bool live = row < g.batch;
    float pre[8], bias[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const bool in = live && n1 + e < g.N;
        const int64_t q = (int64_t)row * g.N + n1 + e;
        bias[e] = KIND != kBackward && in ? __ldg(g.bias + n1 + e) : 0.f;
        pre[e] = KIND == kForward || !in || !g.train ? 0.f : KIND == kOutput ? __ldg(g.y + q) : __ldg(g.z + q);
    }
    bool ok = tile_wait(t.ld, g.st);
    if (ok) ok = tile_mma(t, sa, sb, g.Kp, g.st);
    if (ok) {
        float sq = 0.f;
        float v[8];
        tile_read(t, v);
        __nv_bfloat16 o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int n = n1 + e;
            const int64_t q = (int64_t)row * g.N + n;
            float a = 0.f;
            if (live && n < g.N) {
                if (KIND == kForward) {
                    const float z = v[e] + bias[e];
                    if (g.train) g.z[q] = z;
                    a = gelu(z);
                } else if (KIND == kOutput) {
                    const float z = v[e] + bias[e];
                    g.zo[q] = z;
                    if (g.train) {
                        const float d = z - pre[e];
                        sq += d * d;
                        a = 2.f * d * g.scale;
                        g.dz[q] = a;
                    }
                } else {
                    a = v[e] * gelu_grad(pre[e]);
                    g.dz[q] = a;
                }
            }
            o[e] = __float2bfloat16(a);
        }
        if (g.out) *reinterpret_cast<uint4*>(g.out + img(row, n1, g.outK)) = *reinterpret_cast<const uint4*>(o);
        if (g.outT && row < g.Bp)
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (n1 + e < g.N) g.outT[img(n1 + e, row, g.Bp)] = o[e];
        if (KIND == kOutput && g.train) {
            for (int off = 16; off > 0; off >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, off);
            if ((tid & 31) == 0) g.loss[(blockIdx.y * gridDim.x + blockIdx.x) * (LT / 32) + (tid >> 5)] = sq;
        }
    }
    tile_end(t);
}

// One weight matrix: dW [M][N] = dZ^T A, K along the batch.
struct WeightGrad {
    const __nv_bfloat16 *dzT, *aT;  // images [M][Bp], [N][Bp]
    const float* dz;                // [batch][M]: the bias gradient's terms
    int M, N, tiles_n, first;       // first CTA
    int64_t oW, ob;                 // of the weights and biases in the parameter vector
};
struct WeightArgs {
    WeightGrad w[3];
    int batch, Bp, nloss;
    const float* loss_part;
    volatile float* loss;  // mapped
    float* g;
    Status st;
};

// One block per SM: registers for 32 loads of the bias sums in flight (without it
// the compiler takes 32 registers and a step at a batch of 512 11 us more).
__global__ void __launch_bounds__(LT, 1) k_weights(const __grid_constant__ WeightArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ Tile t;
    const int tid = threadIdx.x;
    const int l = blockIdx.x >= (unsigned)a.w[2].first ? 2 : blockIdx.x >= (unsigned)a.w[1].first ? 1 : 0;
    const WeightGrad& w = a.w[l];
    const int tile = blockIdx.x - w.first, m0 = tile / w.tiles_n * LM, n0 = tile % w.tiles_n * LN;
    uint8_t *sa = smem, *sb = smem + LM * a.Bp * 2;
    tile_begin(t);
    dep_launch();
    dep_wait();
    if (tid == 0) {
        tile_expect(t, (LM + LN) * a.Bp * 2);
        tile_copy(t, sa, w.dzT + img(m0, 0, a.Bp), LM * a.Bp * 2);
        tile_copy(t, sb, w.aT + img(n0, 0, a.Bp), LN * a.Bp * 2);
    }
    // bias gradient of feature mb, by the threads that issue nothing
    const int mb = m0 + tid - LM;
    const bool bias = n0 == 0 && tid >= LM && mb < w.M;
    float db = 0.f;
    if (bias) {
        const float* __restrict__ dz = w.dz + mb;
#pragma unroll 32
        for (int b = 0; b < a.batch; ++b) db += __ldg(dz + (int64_t)b * w.M);
    }
    bool ok = tile_wait(t.ld, a.st);
    if (ok) ok = tile_mma(t, sa, sb, a.Bp, a.st);
    if (ok) {
        // through shared memory (the operand tiles are done with), so that the
        // gradients are written along their rows
        float* c = reinterpret_cast<float*>(smem);
        {
            float v[8];
            tile_read(t, v);
#pragma unroll
            for (int e = 0; e < 8; ++e) c[tile_row() * (LN + 1) + tile_col() + e] = v[e];
        }
        __syncthreads();
        const int n = n0 + (tid & (LN - 1));
        constexpr int kRows = LM * LN / LT;  // rows of this thread: tid / 16, + 16, ...
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int r = tid / LN + i * (LT / LN), m = m0 + r;
            if (m < w.M && n < w.N) a.g[w.oW + (int64_t)m * w.N + n] = c[r * (LN + 1) + (tid & (LN - 1))];
        }
        if (bias) a.g[w.ob + mb] = db;
        if (blockIdx.x == 0 && tid == 0) {
            float s = 0.f;
            for (int i = 0; i < a.nloss; ++i) s += a.loss_part[i];
            *a.loss = s;
        }
    }
    tile_end(t);
}

// AdamW on all parameters, and the images of the stepped weights.
struct StepWeights {
    int64_t oW;  // weights [M][N] in the parameter vector
    int M, N;
    __nv_bfloat16 *im, *imT;  // images [M][Kp], [N][KpT] (imT may be null)
    int Kp, KpT;
};
struct StepArgs {
    StepWeights w[3];
    int64_t np;
    const float* g;
    float *p, *m, *v;
    __nv_bfloat16* pb;
    float lr, b1, b2, eps, wd, c1, c2;
    Status st;
};

// k_adamw's operations with its fused multiply-adds written out, so that both
// train to the same bits
__global__ void __launch_bounds__(LT) k_step(const __grid_constant__ StepArgs a) {
    dep_wait();
    if (*a.st.dev == a.st.gen) return;  // every kernel that could set it has ended
    for (int64_t q = blockIdx.x * LT + threadIdx.x; q < a.np; q += (int64_t)gridDim.x * LT) {
        const float gq = a.g[q], w = a.p[q];
        const float mq = fmaf(1.f - a.b1, gq, __fmul_rn(a.b1, a.m[q]));
        const float vq = fmaf(__fmul_rn(1.f - a.b2, gq), gq, __fmul_rn(a.b2, a.v[q]));
        a.m[q] = mq;
        a.v[q] = vq;
        const float r = fmaf(-a.lr, fmaf(a.wd, w, (mq / a.c1) / (sqrtf(vq / a.c2) + a.eps)), w);
        a.p[q] = r;
        const __nv_bfloat16 h = __float2bfloat16(r);
        a.pb[q] = h;
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            const StepWeights& s = a.w[l];
            if (q < s.oW || q >= s.oW + (int64_t)s.M * s.N) continue;
            const int e = (int)(q - s.oW), m = e / s.N, n = e - m * s.N;
            s.im[img(m, n, s.Kp)] = h;
            if (s.imT) s.imT[img(n, m, s.KpT)] = h;
        }
    }
}

// the weight images of the FP32 parameters
__global__ void k_pack(const float* __restrict__ p, int M, int N, __nv_bfloat16* im, int Kp, __nv_bfloat16* imT, int KpT) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < M * N; q += gridDim.x * blockDim.x) {
        const int m = q / N, n = q - m * N;
        const __nv_bfloat16 h = __float2bfloat16(p[q]);
        im[img(m, n, Kp)] = h;
        if (imT) imT[img(n, m, KpT)] = h;
    }
}

}  // namespace
