// The surrogate of the log-likelihood: a multilayer perceptron (d -> 256 -> 256 -> 256 -> 1, GELU) trained online on
// the likelihood evaluations a sampler makes, with fused BF16 kernels of this library (no counterpart in the
// reference, whose nested sampler trains its own neural bounds in numba, bbarolo/bayesian/nautilus/mlp.py:18-118).
//
// Precision: the weights used by the products and the activations are BF16; products accumulate in FP32 on the
// tensor cores (mma.sync m16n8k16: the layers are small GEMMs, at most a few thousand rows, far from the sizes where
// tcgen05 pipelines pay); pre-activations, gradients, the FP32 master weights and Adam's moments are FP32.
//
// For 128 or 256 hidden units and at most 128 inputs an Adam step is three kernels (k_rows, k_wgrad, k_adam):
// the forward pass and the chain of pre-activation gradients are local to a row, so a pair of CTAs takes 16 rows through all
// the layers with their activations in shared memory, then one launch forms all the weight and bias gradients, one
// adds their partial products and steps. Larger networks take the layers one launch each:
//
// One strided GEMM C[m][j] = sum_t A(m, t) B(t, j) (operands staged through shared memory as BF16 tiles)
// with fused epilogues (bias + GELU for the forward layers, the GELU derivative for the backward chain, plain FP32
// for the weight gradients), the output layer and the loss, column sums for the bias gradients, and Adam.

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "../../include/bbgpu.h"

namespace {

constexpr int GT = 64;       // tile of m and of j
constexpr int GK = 32;       // chunk of t
constexpr int GPAD = 8;      // (padding of the shared-memory rows: no bank conflicts on the fragment loads)
constexpr int KSPLIT = 8;    // K ranges of the weight-gradient products (K = the batch rows)

enum Epi { EPI_BIAS_GELU = 0, EPI_GELU_GRAD = 1, EPI_F32 = 2 };

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// element (i, k) of a strided BF16 operand: p[i * si + k * sk]
__device__ __forceinline__ __nv_bfloat16 elem(const __nv_bfloat16 *p, long long off) { return p[off]; }

// C (M x N) = A (M x K) B (K x N), A(m, t) = A[m sam + t sat], B(t, j) = B[t sbt + j sbj]. Epilogues:
//  EPI_BIAS_GELU: z = C + bias[j] -> Z[m][j] (FP32), out[m][j] = gelu(z) (BF16)
//  EPI_GELU_GRAD: out[m][j] = C * gelu'(Z[m][j]) (BF16, the pre-activation gradient of the layer below), and also
//                 into F32[m][j] when given
//  EPI_F32: F32[m][j] = C (FP32)
// 128 threads: 4 warps of 32 x 32 in a 64 x 64 tile; mma.sync.m16n8k16 row.col BF16 -> FP32.
template <typename TA, typename TB, int EPI>
__global__ void __launch_bounds__(128) k_gemm(int M, int N, int K, const TA *__restrict__ A, long long sam,
                                              long long sat, const TB *__restrict__ B, long long sbt, long long sbj,
                                              const float *__restrict__ bias, float *__restrict__ Z,
                                              __nv_bfloat16 *__restrict__ out, float *__restrict__ F32) {
    __shared__ __align__(16) __nv_bfloat16 As[GT][GK + GPAD];
    __shared__ __align__(16) __nv_bfloat16 Bs[GT][GK + GPAD];   // [j][t]
    const int m0 = blockIdx.y * GT, j0 = blockIdx.x * GT;
    // split K (EPI_F32 only): block z takes the K range [z kper, (z + 1) kper) and writes its partial product to
    // F32 + z M N (summed in order by k_sum_splits)
    const int kper = (K + gridDim.z - 1) / gridDim.z;
    const int tb = blockIdx.z * kper, te = min(K, tb + kper);
    if (EPI == EPI_F32) F32 += (size_t)blockIdx.z * M * N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp >> 1) * 32, wj = (warp & 1) * 32;
    const int g = lane >> 2, c = lane & 3;
    float acc[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[a][b][q] = 0.0f;
    for (int t0 = tb; t0 < te; t0 += GK) {
        for (int e = threadIdx.x; e < GT * GK; e += 128) {
            const int i = e / GK, t = e % GK;
            const int m = m0 + i, j = j0 + i, tt = t0 + t;
            As[i][t] = (m < M && tt < te) ? elem(A, (long long)m * sam + (long long)tt * sat)
                                          : __float2bfloat16_rn(0.0f);
            Bs[i][t] = (j < N && tt < te) ? elem(B, (long long)tt * sbt + (long long)j * sbj)
                                          : __float2bfloat16_rn(0.0f);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GK; kk += 16) {
            uint32_t af[2][4], bf[4][2];
#pragma unroll
            for (int a = 0; a < 2; a++) {
                const int r = wm + a * 16 + g;
                af[a][0] = *(const uint32_t *)&As[r][kk + 2 * c];
                af[a][1] = *(const uint32_t *)&As[r + 8][kk + 2 * c];
                af[a][2] = *(const uint32_t *)&As[r][kk + 2 * c + 8];
                af[a][3] = *(const uint32_t *)&As[r + 8][kk + 2 * c + 8];
            }
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int n = wj + b * 8 + g;
                bf[b][0] = *(const uint32_t *)&Bs[n][kk + 2 * c];
                bf[b][1] = *(const uint32_t *)&Bs[n][kk + 2 * c + 8];
            }
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
                for (int b = 0; b < 4; b++)
                    asm volatile(
                        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
                        "{%8,%9}, {%0,%1,%2,%3};"
                        : "+f"(acc[a][b][0]), "+f"(acc[a][b][1]), "+f"(acc[a][b][2]), "+f"(acc[a][b][3])
                        : "r"(af[a][0]), "r"(af[a][1]), "r"(af[a][2]), "r"(af[a][3]), "r"(bf[b][0]), "r"(bf[b][1]));
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int m = m0 + wm + a * 16 + g + (q >= 2 ? 8 : 0);
                const int j = j0 + wj + b * 8 + 2 * c + (q & 1);
                if (m >= M || j >= N) continue;
                const size_t o = (size_t)m * N + j;
                const float v = acc[a][b][q];
                if (EPI == EPI_BIAS_GELU) {
                    const float z = v + bias[j];
                    Z[o] = z;
                    out[o] = __float2bfloat16_rn(gelu(z));
                } else if (EPI == EPI_GELU_GRAD) {
                    const float d = v * gelu_grad(Z[o]);
                    out[o] = __float2bfloat16_rn(d);
                    if (F32) F32[o] = d;
                } else {
                    F32[o] = v;
                }
            }
}

// the output layer and the loss: y[b] = a[b] . w + bias (warp per row); with targets, r = y - t, dy = 2 r / n (the
// gradient of the mean squared error) and the loss sum of r^2 into loss[0] (atomic)
__global__ void k_output(int n, int H, const __nv_bfloat16 *__restrict__ a, const __nv_bfloat16 *__restrict__ w,
                         const float *__restrict__ bias, const float *__restrict__ t, float *__restrict__ y,
                         float *__restrict__ dy, float *__restrict__ loss) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= n) return;
    float s = 0.0f;
    for (int k = lane; k < H; k += 32) s += __bfloat162float(a[(size_t)row * H + k]) * __bfloat162float(w[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        const float v = s + bias[0];
        y[row] = v;
        if (t) {
            const float r = v - t[row];
            dy[row] = 2.0f * r / (float)n;
            atomicAdd(loss, r * r);
        }
    }
}

// the gradient of the last hidden layer's pre-activation: dz[b][k] = dy[b] w[k] gelu'(z[b][k]) (BF16)
__global__ void k_out_back(int n, int H, const float *__restrict__ dy, const __nv_bfloat16 *__restrict__ w,
                           const float *__restrict__ z, __nv_bfloat16 *__restrict__ dz, float *__restrict__ dz32) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)n * H) return;
    const int b = (int)(i / H), k = (int)(i % H);
    const float d = dy[b] * __bfloat162float(w[k]) * gelu_grad(z[i]);
    dz[i] = __float2bfloat16_rn(d);
    if (dz32) dz32[i] = d;
}

// column sums: out[j] = sum_b in[b][j] (or, with v given, sum_b v[b] a[b][j]: the output weights' gradient); a block
// of 32 columns x 32 row groups, the groups' partial sums added in shared memory
__global__ void __launch_bounds__(1024) k_colsum(int n, int N, const float *__restrict__ in,
                                                 const float *__restrict__ v, const __nv_bfloat16 *__restrict__ a,
                                                 float *__restrict__ out) {
    __shared__ float part[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + tx;
    float s = 0.0f;
    if (j < N)
        for (int b = ty; b < n; b += 32)
            s += v ? v[b] * __bfloat162float(a[(size_t)b * N + j]) : in[(size_t)b * N + j];
    part[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && j < N) {
        float t = 0.0f;
        for (int k = 0; k < 32; k++) t += part[k][tx];
        out[j] = t;
    }
}

// out[i] = sum over the splits z (in order) of part[z][i]
__global__ void k_sum_splits(long long n, int nsplit, const float *__restrict__ part, float *__restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float a = part[i];
    for (int z = 1; z < nsplit; z++) a += part[(size_t)z * n + i];
    out[i] = a;
}

__global__ void k_sum(int n, const float *__restrict__ v, float *__restrict__ out) {
    __shared__ float sh[256];
    float s = 0.0f;
    for (int i = threadIdx.x; i < n; i += 256) s += v[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int d = 128; d > 0; d >>= 1) {
        if (threadIdx.x < d) sh[threadIdx.x] += sh[threadIdx.x + d];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = sh[0];
}

// ---------------------------------------------------------------------- networks of at most 256 hidden units
// What bounds these kernels is latency: a step of 1024 rows and 8 x 256 x 256 x 256 weights is 0.8 GFLOP, but it was 21
// launches of GEMMs whose 2-byte loads took 22-31 us each (219 us a step); the three launches take 40. All sums keep
// the order of the layer-by-layer path (mma.sync over K in steps of 16, the same splits of the batch), so the weights
// are the same bit for bit.
constexpr int RB = 16;          // rows of a CTA of k_rows (one mma tile)
constexpr int RT = 256;         // its threads
constexpr int RSTAGE = 6;       // stages of 32 weight rows or columns in flight
constexpr int MAXD = 128;

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s32(dst)), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s32(p)));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s32(p)));
}
__device__ __forceinline__ void ldm2(uint32_t (&r)[2], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(s32(p)));
}
__device__ __forceinline__ void ldm2t(uint32_t (&r)[2], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1]) : "r"(s32(p)));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// row r of step `step`'s minibatch in the training set
__device__ __forceinline__ long long batch_row(unsigned long long seed, int step, int r, int n) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * ((unsigned long long)step * 0x100000001ull + r + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (long long)(z % (unsigned long long)n);
}

struct RowsArgs {
    int n, d, back, setn, step;       // rows, inputs; the backward chain too; rows of the training set (0: x has the rows)
    unsigned long long seed;
    const float *x, *ts;              // inputs (n x d, or the set's) and targets (or the set's)
    const __nv_bfloat16 *w16;
    const float *w;
    long long off[8];
    __nv_bfloat16 *xp, *a[3], *dz[3]; // inputs (n x round16(d)), activations, pre-activation gradients (n x H)
    float *dz32[3], *y, *dy, *r2;     // the gradients in FP32; outputs, their gradients, squared residuals
};

// H = 128 NT. A cluster of two CTAs takes 16 rows, each half of every layer's columns (warp w of CTA q the columns
// H/2 q + 8 NT w ..): a single CTA streamed all the weights (36 us a step of 1024 rows on 64 SMs against 28). The
// weights come through a ring of 32-deep slices, the next layer's behind the last one's; a layer's outputs are written
// to both CTAs' shared memory.
template <int NT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(RT) k_rows(RowsArgs A) {
    constexpr int H = 128 * NT, HH = H / 2, HP = H + 8, BP = HH + 8;
    constexpr int SLICE = (HH * 40 > 32 * BP ? HH * 40 : 32 * BP);           // elements of a stage
    extern __shared__ __align__(16) uint8_t rsm[];
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int half = (int)cl.block_rank(), h0 = half * HH;
    const int d = A.d, dp = (d + 15) & ~15, kx = (d + 31) / 32;
    __nv_bfloat16 *const ring = (__nv_bfloat16 *)rsm;
    __nv_bfloat16 *const xs = ring + RSTAGE * SLICE;                         // RB x (32 kx + 8)
    const int xpitch = 32 * kx + 8;
    __nv_bfloat16 *const act = xs + RB * (MAXD + 8);                         // 3 x RB x HP; then the gradients
    __nv_bfloat16 *const peer = cl.map_shared_rank(act, half ^ 1);
    float *const Z = (float *)(act + 3 * RB * HP), *const E = Z + 3 * RB * HH;   // 3 x RB x HH: z, erf(z / sqrt 2)
    __shared__ float sdy[RB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int r0 = (blockIdx.x >> 1) * RB, rows = min(RB, A.n - r0);
    // slice q of the stream: the first layer's kx, then H / 32 of layers 2 and 3, then of layers 3 and 2 backwards
    constexpr int KH = H / 32;
    const int nq = kx + (A.back ? 4 : 2) * KH;
    auto issue = [&](int q) {
        if (q < nq) {
            __nv_bfloat16 *st = ring + (q % RSTAGE) * SLICE;
            if (q < kx) {                                                    // (rows of d inputs: not aligned)
                const __nv_bfloat16 *W = A.w16 + A.off[0] + (size_t)h0 * d;
                for (int e = tid; e < HH * 32; e += RT) {
                    const int j = e >> 5, t = q * 32 + (e & 31);
                    st[j * 40 + (e & 31)] = t < d ? W[(size_t)j * d + t] : __float2bfloat16_rn(0.0f);
                }
            } else {
                const int l = (q - kx) / KH, k = (q - kx) % KH;              // 0, 1: layers 2, 3; 2, 3: back 3, 2
                const __nv_bfloat16 *W = A.w16 + A.off[l == 0 || l == 3 ? 2 : 4];
                if (l < 2)
                    for (int e = tid; e < HH * 4; e += RT)
                        cp16(st + (e >> 2) * 40 + (e & 3) * 8, W + (size_t)(h0 + (e >> 2)) * H + k * 32 + (e & 3) * 8);
                else
                    for (int e = tid; e < 32 * (HH / 8); e += RT)
                        cp16(st + (e / (HH / 8)) * BP + (e % (HH / 8)) * 8,
                             W + (size_t)(k * 32 + e / (HH / 8)) * H + h0 + (e % (HH / 8)) * 8);
            }
        }
        cp_commit();
    };
    for (int q = 0; q < RSTAGE - 1; q++) issue(q);
    // the rows' inputs in BF16, zero beyond d and n
    for (int e = tid; e < RB * 32 * kx; e += RT) {
        const int r = e / (32 * kx), k = e % (32 * kx);
        float v = 0.0f;
        if (r < rows && k < d)
            v = A.x[(size_t)(A.setn ? batch_row(A.seed, A.step, r0 + r, A.setn) : r0 + r) * d + k];
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        xs[r * xpitch + k] = h;
        if (A.back && half == 0 && r < rows && k < dp) A.xp[(size_t)(r0 + r) * dp + k] = h;
    }
    float acc[NT][4];
    int q = 0;
    // C (16 x H / 2) = A (16 x 32 nk, pitch ap) B, slices q .. q + nk
    auto product = [&](const __nv_bfloat16 *a, int ap, int nk, bool back) {
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
        for (int k = 0; k < nk; k++, q++) {
            cp_wait<RSTAGE - 2>();
            __syncthreads();
            issue(q + RSTAGE - 1);
            const __nv_bfloat16 *st = ring + (q % RSTAGE) * SLICE;
#pragma unroll
            for (int kk = 0; kk < 32; kk += 16) {
                uint32_t af[4];
                ldm4(af, a + (lane & 15) * ap + k * 32 + kk + (lane >> 4) * 8);
#pragma unroll
                for (int i = 0; i < NT; i++) {
                    const int n0 = (warp * NT + i) * 8;
                    uint32_t bf[2];
                    if (!back) ldm2(bf, st + (n0 + (lane & 7)) * 40 + kk + ((lane >> 3) & 1) * 8);
                    else ldm2t(bf, st + (kk + (lane & 15)) * BP + n0);
                    mma16816(acc[i], af, bf);
                }
            }
        }
    };
    // two neighbouring values of row r, columns h0 + col, col + 1 of slot l, into both CTAs' activations
    auto put = [&](int l, int r, int col, float v0, float v1) {
        const __nv_bfloat162 v{__float2bfloat16_rn(v0), __float2bfloat16_rn(v1)};
        const int o = (l * RB + r) * HP + h0 + col;
        *(__nv_bfloat162 *)(act + o) = v;
        *(__nv_bfloat162 *)(peer + o) = v;
    };
    // this CTA's rows of slot l to global memory
    auto store = [&](int l, __nv_bfloat16 *out) {
        for (int e = tid; e < rows * (HH / 8); e += RT) {
            const int r = e / (HH / 8), k = h0 + (e % (HH / 8)) * 8;
            *(uint4 *)(out + (size_t)(r0 + r) * H + k) = *(const uint4 *)(act + (l * RB + r) * HP + k);
        }
    };
    cl.sync();                                              // (the peer is running before its memory is written)
    for (int l = 0; l < 3; l++) {
        if (l == 0) product(xs, xpitch, kx, false);
        else product(act + (l - 1) * RB * HP, HP, KH, false);
        const float *bias = A.w + A.off[2 * l + 1] + h0;
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int r = g + (j >= 2 ? 8 : 0), col = (warp * NT + i) * 8 + 2 * c;
                float a2[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const float z = acc[i][j + u] + bias[col + u], e = erff(z * 0.70710678118654752f);
                    Z[(l * RB + r) * HH + col + u] = z;
                    E[(l * RB + r) * HH + col + u] = e;
                    a2[u] = 0.5f * z * (1.0f + e);          // gelu
                }
                put(l, r, col, a2[0], a2[1]);
            }
        cl.sync();
        if (A.back) store(l, A.a[l]);
    }
    // the output and, with the backward chain, its gradient (mean squared error)
    const __nv_bfloat16 *w4 = A.w16 + A.off[6];
    for (int r = warp; r < rows; r += RT / 32) {
        const __nv_bfloat16 *a = act + (2 * RB + r) * HP;
        float v = 0.0f;
        for (int k = lane; k < H; k += 32) v += __bfloat162float(a[k]) * __bfloat162float(w4[k]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) {
            v += A.w[A.off[7]];
            if (half == 0) A.y[r0 + r] = v;
            if (A.back) {
                const float t = A.ts[A.setn ? batch_row(A.seed, A.step, r0 + r, A.setn) : r0 + r];
                const float e = v - t;
                sdy[r] = 2.0f * e / (float)A.n;
                if (half == 0) {
                    A.dy[r0 + r] = sdy[r];
                    A.r2[r0 + r] = e * e;
                }
            }
        }
    }
    cl.sync();                                              // (both CTAs have read the last activations)
    if (!A.back) return;
    // the pre-activation gradients take the activations' place, layer 3 in slot 2 and so on down
    auto dgelu = [&](int l, int r, int col) {
        const float z = Z[(l * RB + r) * HH + col];
        return 0.5f * (1.0f + E[(l * RB + r) * HH + col]) + z * 0.39894228040143268f * expf(-0.5f * z * z);
    };
    for (int e = tid; e < RB * (HH / 2); e += RT) {
        const int r = e / (HH / 2), k = e % (HH / 2) * 2;
        float v[2] = {0.0f, 0.0f};
        if (r < rows) {
#pragma unroll
            for (int u = 0; u < 2; u++) v[u] = sdy[r] * __bfloat162float(w4[h0 + k + u]) * dgelu(2, r, k + u);
            *(float2 *)(A.dz32[2] + (size_t)(r0 + r) * H + h0 + k) = make_float2(v[0], v[1]);
        }
        put(2, r, k, v[0], v[1]);
    }
    cl.sync();
    store(2, A.dz[2]);
    for (int l = 1; l >= 0; l--) {
        product(act + (l + 1) * RB * HP, HP, KH, true);
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const int r = g + (j >= 2 ? 8 : 0), col = (warp * NT + i) * 8 + 2 * c;
                const float v0 = acc[i][j] * dgelu(l, r, col), v1 = acc[i][j + 1] * dgelu(l, r, col + 1);
                put(l, r, col, v0, v1);
                if (r < rows) *(float2 *)(A.dz32[l] + (size_t)(r0 + r) * H + h0 + col) = make_float2(v0, v1);
            }
        cl.sync();
        store(l, A.dz[l]);
    }
}

struct WgradArgs {
    int n, d, dp, H, ns, kper;        // ns ranges of kper rows
    const __nv_bfloat16 *xp, *a[3], *dz[3];
    const float *dz32[3], *dy;
    float *part[3], *gb[3], *gw4, *gb4;
};

// All the gradients that sum over the batch: blocks of 64 x 64 weights of a layer and a range of rows (their partial
// products to part[l] + z H kin), then blocks of 8 columns of the bias and output-weight sums, then the output bias.
constexpr int WCH = 32;         // rows of a slice
constexpr int WST = 4;          // slices in flight
__global__ void __launch_bounds__(128) k_wgrad(WgradArgs A) {
    __shared__ __align__(16) __nv_bfloat16 sa[WST][WCH][72], sb[WST][WCH][72];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const int tm = A.H / 64, t12 = tm * tm * A.ns, t0 = tm * ((A.dp + 63) / 64) * A.ns;
    int b = blockIdx.x;
    if (b < 2 * t12 + t0) {
        int l = 2;
        if (b >= t12) {
            b -= t12;
            l = 1;
            if (b >= t12) {
                b -= t12;
                l = 0;
            }
        }
        const int kin = l ? A.H : A.d, kp = l ? A.H : A.dp, tn = l ? tm : (A.dp + 63) / 64;
        const int z = b / (tm * tn), m0 = b % (tm * tn) / tn * 64, j0 = b % tn * 64;
        const __nv_bfloat16 *below = l ? A.a[l - 1] : A.xp, *up = A.dz[l];
        const int tb = z * A.kper, te = min(A.n, tb + A.kper), nk = (te - tb + WCH - 1) / WCH;
        const int wm = (warp >> 1) * 32, wj = (warp & 1) * 32;
        float acc[2][4][4] = {};
        auto issue = [&](int k) {
            if (k < nk)
                for (int e = tid; e < WCH * 8; e += 128) {
                    const int r = e >> 3, o = (e & 7) * 8, row = tb + k * WCH + r;
                    if (row < te) cp16(&sa[k % WST][r][o], up + (size_t)row * A.H + m0 + o);
                    else *(uint4 *)&sa[k % WST][r][o] = make_uint4(0, 0, 0, 0);
                    if (row < te && j0 + o < kp) cp16(&sb[k % WST][r][o], below + (size_t)row * kp + j0 + o);
                    else *(uint4 *)&sb[k % WST][r][o] = make_uint4(0, 0, 0, 0);
                }
            cp_commit();
        };
        for (int k = 0; k < WST - 1; k++) issue(k);
        for (int k = 0; k < nk; k++) {
            cp_wait<WST - 2>();
            __syncthreads();
            issue(k + WST - 1);
#pragma unroll
            for (int kk = 0; kk < WCH; kk += 16) {
                uint32_t af[2][4], bf[2];
#pragma unroll
                for (int i = 0; i < 2; i++)
                    ldm4t(af[i], &sa[k % WST][kk + (lane >> 4) * 8 + (lane & 7)][wm + i * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    ldm2t(bf, &sb[k % WST][kk + (lane & 15)][wj + j * 8]);
#pragma unroll
                    for (int i = 0; i < 2; i++) mma16816(acc[i][j], af[i], bf);
                }
            }
        }
        float *P = A.part[l] + (size_t)z * A.H * kin;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int m = m0 + wm + i * 16 + g + (q >= 2 ? 8 : 0), n = j0 + wj + j * 8 + 2 * c + (q & 1);
                    if (n < kin) P[(size_t)m * kin + n] = acc[i][j][q];
                }
        return;
    }
    b -= 2 * t12 + t0;
    float *const part = (float *)sa;                        // 32 x 9
    if (b < 4 * (A.H / 8)) {
        // 8 columns, the rows of each in 32 groups (rows k, k + 32, ...), two a thread; the groups added in order
        const int l = b / (A.H / 8), j = b % (A.H / 8) * 8 + (tid & 7), k0 = tid >> 3;
        float s[2] = {};
        if (l < 3) {
            const float *in = A.dz32[l] + j;
#pragma unroll 8
            for (int r = k0; r < A.n; r += 32) {
                s[0] += in[(size_t)r * A.H];
                s[1] += r + 16 < A.n ? in[(size_t)(r + 16) * A.H] : 0.0f;
            }
        } else {
            const __nv_bfloat16 *in = A.a[2] + j;
#pragma unroll 8
            for (int r = k0; r < A.n; r += 32) {
                s[0] += A.dy[r] * __bfloat162float(in[(size_t)r * A.H]);
                if (r + 16 < A.n) s[1] += A.dy[r + 16] * __bfloat162float(in[(size_t)(r + 16) * A.H]);
            }
        }
        part[k0 * 9 + (tid & 7)] = s[0];
        part[(k0 + 16) * 9 + (tid & 7)] = s[1];
        __syncthreads();
        if (tid < 8) {
            float t = 0.0f;
            for (int k = 0; k < 32; k++) t += part[k * 9 + tid];
            (l < 3 ? A.gb[l] : A.gw4)[j] = t;
        }
        return;
    }
    float s0 = 0.0f, s1 = 0.0f;                             // (k_sum's 256 threads, two a thread)
    for (int i = tid; i < A.n; i += 256) s0 += A.dy[i];
    for (int i = tid + 128; i < A.n; i += 256) s1 += A.dy[i];
    part[tid] = s0 + s1;
    __syncthreads();
    for (int k = 64; k > 0; k >>= 1) {
        if (tid < k) part[tid] += part[tid + k];
        __syncthreads();
    }
    if (tid == 0) A.gb4[0] = part[0];
}

// the weight gradients' partial products added in order, into the gradient
struct SplitArgs {
    long long off[3], size[3];        // the weights W1, W2, W3 in the parameters
    const float *part[3];
    int ns;                           // 0: the gradient is in g
};
__device__ __forceinline__ float split_sum(const SplitArgs &S, long long i, float gi) {
    if (S.ns == 0) return gi;
#pragma unroll
    for (int l = 0; l < 3; l++)
        if (i >= S.off[l] && i < S.off[l] + S.size[l]) {
            const float *p = S.part[l] + (i - S.off[l]);
            float v[KSPLIT];                                // (all loads before the first sum)
#pragma unroll
            for (int z = 0; z < KSPLIT; z++) v[z] = z < S.ns ? p[(size_t)z * S.size[l]] : 0.0f;
            gi = v[0];
#pragma unroll
            for (int z = 1; z < KSPLIT; z++) gi += v[z];
        }
    return gi;
}

__global__ void k_split_sums(long long n, SplitArgs S, float *__restrict__ g) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) g[i] = split_sum(S, i, g[i]);
}

// Adam on the FP32 master weights, the BF16 copy rewritten (b1t, b2t: 1 - beta^t)
__global__ void k_adam(long long n, float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
                       const float *__restrict__ g, SplitArgs S, __nv_bfloat16 *__restrict__ w16, float lr, float b1, float b2,
                       float b1t, float b2t, float eps) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = split_sum(S, i, g[i]);
    const float mi = b1 * m[i] + (1.0f - b1) * gi, vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / b1t) / (sqrtf(vi / b2t) + eps);
    w[i] = wi;
    if (w16) w16[i] = __float2bfloat16_rn(wi);
}

__global__ void k_to_bf16(long long n, const float *__restrict__ in, __nv_bfloat16 *__restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

// a minibatch of `rows` rows drawn with replacement from the n rows of a resident training set: row r of step
// `step` is the set's row hash(seed, step, r) mod n (inputs to BF16, targets as they are)
__global__ void k_gather_batch(int rows, int d, int n, unsigned long long seed, int step,
                               const float *__restrict__ xs, const float *__restrict__ ts,
                               __nv_bfloat16 *__restrict__ x16, float *__restrict__ t) {
    const int r = blockIdx.x;
    const long long src = batch_row(seed, step, r, n);
    for (int k = threadIdx.x; k < d; k += blockDim.x) x16[(size_t)r * d + k] = __float2bfloat16_rn(xs[src * d + k]);
    if (threadIdx.x == 0) t[r] = ts[src];
}

}  // namespace

// ------------------------------------------------------------------------------------------------- host side
struct bbgpu_mlp {
    int device = 0, d = 0, H = 0;
    long long np = 0;                 // parameters: W1 (H x d), b1 (H), W2 (H x H), b2, W3 (H x H), b3, w4 (H), b4
    long long off[8] = {};
    float *w = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;   // FP32 master, gradient, Adam moments
    __nv_bfloat16 *w16 = nullptr;     // BF16 copy used by the products
    int step = 0;
    int cap = 0;                      // rows of the batch buffers
    float *xf = nullptr, *t = nullptr, *y = nullptr, *dy = nullptr, *r2 = nullptr, *loss = nullptr;
    __nv_bfloat16 *x16 = nullptr, *a[3] = {}, *dz[3] = {};
    float *z[3] = {}, *dz32[3] = {};             // (z: of the layer-by-layer path only)
    float *set_x = nullptr, *set_t = nullptr;   // the resident training set of bbgpu_mlp_train
    float *split = nullptr;                      // the partial weight gradients of the split-K products
    long long set_cap = 0;
    cudaStream_t s = nullptr;
};

namespace {

// the networks of the three-kernel step
bool small_net(const bbgpu_mlp *m) { return (m->H == 128 || m->H == 256) && m->d <= MAXD; }

int grow(bbgpu_mlp *m, int n) {
    if (n <= m->cap) return BBGPU_OK;
    cudaFree(m->xf); cudaFree(m->t); cudaFree(m->y); cudaFree(m->dy); cudaFree(m->r2); cudaFree(m->x16);
    for (int i = 0; i < 3; i++) { cudaFree(m->a[i]); cudaFree(m->z[i]); }
    for (int i = 0; i < 3; i++) { cudaFree(m->dz[i]); cudaFree(m->dz32[i]); }
    const bool small = small_net(m);
    const size_t nh = (size_t)n * m->H;
    bool ok = cudaMalloc(&m->xf, sizeof(float) * (size_t)n * m->d) == cudaSuccess &&
              cudaMalloc(&m->x16, sizeof(__nv_bfloat16) * (size_t)n * ((m->d + 15) & ~15)) == cudaSuccess &&
              cudaMalloc(&m->t, sizeof(float) * n) == cudaSuccess && cudaMalloc(&m->y, sizeof(float) * n) == cudaSuccess &&
              cudaMalloc(&m->dy, sizeof(float) * n) == cudaSuccess && cudaMalloc(&m->r2, sizeof(float) * n) == cudaSuccess;
    for (int i = 0; i < 3 && ok; i++)
        ok = cudaMalloc(&m->a[i], sizeof(__nv_bfloat16) * nh) == cudaSuccess &&
             (small || cudaMalloc(&m->z[i], sizeof(float) * nh) == cudaSuccess);
    for (int i = 0; i < (small ? 3 : 2) && ok; i++)
        ok = cudaMalloc(&m->dz[i], sizeof(__nv_bfloat16) * nh) == cudaSuccess &&
             cudaMalloc(&m->dz32[i], sizeof(float) * nh) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        m->cap = 0;
        return BBGPU_ERR_NOMEM;
    }
    m->cap = n;
    return BBGPU_OK;
}

template <typename TA, typename TB, int EPI>
void gemm(cudaStream_t s, int M, int N, int K, const TA *A, long long sam, long long sat, const TB *B, long long sbt,
          long long sbj, const float *bias, float *Z, __nv_bfloat16 *out, float *F32, int nsplit = 1) {
    dim3 grid((N + GT - 1) / GT, (M + GT - 1) / GT, nsplit);
    k_gemm<TA, TB, EPI><<<grid, 128, 0, s>>>(M, N, K, A, sam, sat, B, sbt, sbj, bias, Z, out, F32);
}

// the forward pass of n rows of m->x16 (and with targets t, the loss and dy)
void forward(bbgpu_mlp *m, int n, const float *t) {
    const int d = m->d, H = m->H;
    const __nv_bfloat16 *W = m->w16;
    const float *b = m->w;
    gemm<__nv_bfloat16, __nv_bfloat16, EPI_BIAS_GELU>(m->s, n, H, d, m->x16, d, 1, W + m->off[0], 1, d,
                                                      b + m->off[1], m->z[0], m->a[0], nullptr);
    for (int l = 1; l < 3; l++)
        gemm<__nv_bfloat16, __nv_bfloat16, EPI_BIAS_GELU>(m->s, n, H, H, m->a[l - 1], H, 1, W + m->off[2 * l], 1, H,
                                                          b + m->off[2 * l + 1], m->z[l], m->a[l], nullptr);
    if (t) cudaMemsetAsync(m->loss, 0, sizeof(float), m->s);
    k_output<<<(n + 7) / 8, 256, 0, m->s>>>(n, H, m->a[2], W + m->off[6], b + m->off[7], t, m->y, m->dy, m->loss);
}

// the gradient of the mean squared error over the n rows, into m->g
void backward(bbgpu_mlp *m, int n) {
    const int d = m->d, H = m->H;
    const __nv_bfloat16 *W = m->w16;
    float *G = m->g;
    const size_t nh = (size_t)n * H;
    k_out_back<<<(unsigned)((nh + 255) / 256), 256, 0, m->s>>>(n, H, m->dy, W + m->off[6], m->z[2], m->dz[0],
                                                                m->dz32[0]);
    k_colsum<<<(H + 31) / 32, 1024, 0, m->s>>>(n, H, nullptr, m->dy, m->a[2], G + m->off[6]);
    k_sum<<<1, 256, 0, m->s>>>(n, m->dy, G + m->off[7]);
    int cur = 0;
    for (int l = 2; l >= 0; l--) {
        const __nv_bfloat16 *below = l > 0 ? m->a[l - 1] : m->x16;
        const int kin = l > 0 ? H : d;
        // weight gradient: G[j][k] = sum_b dz[b][j] below[b][k]; bias gradient: column sums of dz
        // (K = the batch rows: split in KSPLIT ranges, the partial products summed in order)
        const int ns = std::max(1, std::min(KSPLIT, n / 128));
        gemm<__nv_bfloat16, __nv_bfloat16, EPI_F32>(m->s, H, kin, n, m->dz[cur], 1, H, below, kin, 1, nullptr,
                                                    nullptr, nullptr, ns > 1 ? m->split : G + m->off[2 * l], ns);
        if (ns > 1) {
            const long long nn = (long long)H * kin;
            k_sum_splits<<<(unsigned)((nn + 255) / 256), 256, 0, m->s>>>(nn, ns, m->split, G + m->off[2 * l]);
        }
        k_colsum<<<(H + 31) / 32, 1024, 0, m->s>>>(n, H, m->dz32[cur], nullptr, nullptr, G + m->off[2 * l + 1]);
        if (l > 0)   // the layer below: dz'[b][k] = (sum_j dz[b][j] W[j][k]) gelu'(z'[b][k])
            gemm<__nv_bfloat16, __nv_bfloat16, EPI_GELU_GRAD>(m->s, n, H, H, m->dz[cur], H, 1, W + m->off[2 * l], H,
                                                              1, nullptr, m->z[l - 1], m->dz[1 - cur],
                                                              m->dz32[1 - cur]);
        cur = 1 - cur;
    }
}

// the rows of x (or, with setn, step `step`'s minibatch of the set x, t) through the network: y; with t also the loss
// terms and the chain of gradients
int rows_pass(bbgpu_mlp *m, const float *x, const float *t, int n, int setn, int step, uint64_t seed) {
    RowsArgs A{};
    A.n = n;
    A.d = m->d;
    A.back = t ? 1 : 0;
    A.setn = setn;
    A.step = step;
    A.seed = seed;
    A.x = x;
    A.ts = t;
    A.w16 = m->w16;
    A.w = m->w;
    memcpy(A.off, m->off, sizeof A.off);
    A.xp = m->x16;
    for (int i = 0; i < 3; i++) {
        A.a[i] = m->a[i];
        A.dz[i] = m->dz[i];
        A.dz32[i] = m->dz32[i];
    }
    A.y = m->y;
    A.dy = m->dy;
    A.r2 = m->r2;
    auto go = [&](auto kernel, int H) {
        const int HH = H / 2, slice = std::max(HH * 40, 32 * (HH + 8));
        const int smem = 2 * (RSTAGE * slice + RB * (MAXD + 8) + 3 * RB * (H + 8)) + 4 * 6 * RB * HH;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        kernel<<<2 * ((n + RB - 1) / RB), RT, smem, m->s>>>(A);
    };
    if (m->H == 128) go(k_rows<1>, 128);
    else go(k_rows<2>, 256);
    return BBGPU_OK;
}

// the gradients of the rows of rows_pass: biases and output weights into g, the others as partial products
SplitArgs wgrad_pass(bbgpu_mlp *m, int n) {
    WgradArgs A{};
    SplitArgs S{};
    A.n = n;
    A.d = m->d;
    A.dp = (m->d + 15) & ~15;
    A.H = m->H;
    A.ns = std::max(1, std::min(KSPLIT, n / 128));
    A.kper = (n + A.ns - 1) / A.ns;
    A.xp = m->x16;
    S.ns = A.ns;
    float *p = m->split;
    for (int l = 0; l < 3; l++) {
        A.a[l] = m->a[l];
        A.dz[l] = m->dz[l];
        A.dz32[l] = m->dz32[l];
        A.part[l] = p;
        A.gb[l] = m->g + m->off[2 * l + 1];
        S.off[l] = m->off[2 * l];
        S.size[l] = m->off[2 * l + 1] - m->off[2 * l];
        S.part[l] = p;
        p += (size_t)A.ns * S.size[l];
    }
    A.dy = m->dy;
    A.gw4 = m->g + m->off[6];
    A.gb4 = m->g + m->off[7];
    const int tm = m->H / 64;
    k_wgrad<<<(2 * tm * tm + tm * ((A.dp + 63) / 64)) * A.ns + 4 * (m->H / 8) + 1, 128, 0, m->s>>>(A);
    return S;
}

int load_x(bbgpu_mlp *m, const float *x, int n) {
    int rc = grow(m, n);
    if (rc) return rc;
    const size_t nx = (size_t)n * m->d;
    if (cudaMemcpyAsync(m->xf, x, sizeof(float) * nx, cudaMemcpyHostToDevice, m->s) != cudaSuccess)
        return BBGPU_ERR_CUDA;
    if (!small_net(m)) k_to_bf16<<<(unsigned)((nx + 255) / 256), 256, 0, m->s>>>((long long)nx, m->xf, m->x16);
    return BBGPU_OK;
}

int finish(bbgpu_mlp *m) {
    cudaError_t e = cudaStreamSynchronize(m->s);
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? BBGPU_OK : BBGPU_ERR_CUDA;
}

uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace

extern "C" int bbgpu_mlp_create(bbgpu_mlp **out, int device, int d_in, int hidden, uint64_t seed) {
    if (!out || d_in < 1 || d_in > 4096 || hidden < 8 || hidden > 4096) return BBGPU_ERR_ARG;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return BBGPU_ERR_CUDA;
    bbgpu_mlp *m = new bbgpu_mlp();
    m->device = device;
    m->d = d_in;
    m->H = hidden;
    const long long H = hidden, d = d_in;
    const long long sizes[8] = {H * d, H, H * H, H, H * H, H, H, 1};
    for (int i = 0; i < 8; i++) {
        m->off[i] = m->np;
        m->np += sizes[i];
    }
    // initial weights uniform in +-1/sqrt(fan in), biases zero
    std::vector<float> w(m->np, 0.0f);
    const long long fan[4] = {d, H, H, H};
    for (int l = 0; l < 4; l++) {
        const float a = 1.0f / sqrtf((float)fan[l]);
        for (long long i = 0; i < sizes[2 * l]; i++)
            w[m->off[2 * l] + i] = a * (2.0f * (float)((splitmix(seed) >> 11) * (1.0 / 9007199254740992.0)) - 1.0f);
    }
    bool ok = cudaStreamCreateWithFlags(&m->s, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&m->w, sizeof(float) * m->np) == cudaSuccess &&
              cudaMalloc(&m->g, sizeof(float) * m->np) == cudaSuccess &&
              cudaMalloc(&m->m1, sizeof(float) * m->np) == cudaSuccess &&
              cudaMalloc(&m->m2, sizeof(float) * m->np) == cudaSuccess &&
              cudaMalloc(&m->w16, sizeof(__nv_bfloat16) * m->np) == cudaSuccess &&
              cudaMalloc(&m->split, sizeof(float) * KSPLIT * (small_net(m) ? (size_t)m->np : (size_t)hidden * std::max(hidden, d_in))) == cudaSuccess &&
              cudaMalloc(&m->loss, sizeof(float)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        bbgpu_mlp_destroy(m);
        return BBGPU_ERR_NOMEM;
    }
    int rc = bbgpu_mlp_set_params(m, w.data());
    if (rc) {
        bbgpu_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return BBGPU_OK;
}

extern "C" int bbgpu_mlp_destroy(bbgpu_mlp *m) {
    if (!m) return BBGPU_ERR_ARG;
    cudaSetDevice(m->device);
    cudaFree(m->w); cudaFree(m->g); cudaFree(m->m1); cudaFree(m->m2); cudaFree(m->w16); cudaFree(m->loss);
    cudaFree(m->xf); cudaFree(m->t); cudaFree(m->y); cudaFree(m->dy); cudaFree(m->r2); cudaFree(m->x16);
    for (int i = 0; i < 3; i++) { cudaFree(m->a[i]); cudaFree(m->z[i]); }
    for (int i = 0; i < 3; i++) { cudaFree(m->dz[i]); cudaFree(m->dz32[i]); }
    cudaFree(m->set_x); cudaFree(m->set_t); cudaFree(m->split);
    if (m->s) cudaStreamDestroy(m->s);
    delete m;
    return BBGPU_OK;
}

extern "C" long long bbgpu_mlp_nparams(const bbgpu_mlp *m) { return m ? m->np : 0; }

extern "C" int bbgpu_mlp_set_params(bbgpu_mlp *m, const float *p) {
    if (!m || !p) return BBGPU_ERR_ARG;
    if (cudaSetDevice(m->device) != cudaSuccess) return BBGPU_ERR_CUDA;
    cudaMemcpyAsync(m->w, p, sizeof(float) * m->np, cudaMemcpyHostToDevice, m->s);
    cudaMemsetAsync(m->m1, 0, sizeof(float) * m->np, m->s);
    cudaMemsetAsync(m->m2, 0, sizeof(float) * m->np, m->s);
    k_to_bf16<<<(unsigned)((m->np + 255) / 256), 256, 0, m->s>>>(m->np, m->w, m->w16);
    m->step = 0;
    return finish(m);
}

extern "C" int bbgpu_mlp_get_params(const bbgpu_mlp *m, float *p) {
    if (!m || !p) return BBGPU_ERR_ARG;
    if (cudaSetDevice(m->device) != cudaSuccess) return BBGPU_ERR_CUDA;
    return cudaMemcpy(p, m->w, sizeof(float) * m->np, cudaMemcpyDeviceToHost) == cudaSuccess ? BBGPU_OK
                                                                                             : BBGPU_ERR_CUDA;
}

extern "C" int bbgpu_mlp_predict(bbgpu_mlp *m, const float *x, int n, float *y) {
    if (!m || (!x && n) || (!y && n) || n < 0) return BBGPU_ERR_ARG;
    if (n == 0) return BBGPU_OK;
    if (cudaSetDevice(m->device) != cudaSuccess) return BBGPU_ERR_CUDA;
    int rc = load_x(m, x, n);
    if (rc) return rc;
    if (small_net(m)) rows_pass(m, m->xf, nullptr, n, 0, 0, 0);
    else forward(m, n, nullptr);
    cudaMemcpyAsync(y, m->y, sizeof(float) * n, cudaMemcpyDeviceToHost, m->s);
    return finish(m);
}

extern "C" int bbgpu_mlp_gradients(bbgpu_mlp *m, const float *x, const float *t, int n, float *grads, float *loss) {
    if (!m || !x || !t || n < 1) return BBGPU_ERR_ARG;
    if (cudaSetDevice(m->device) != cudaSuccess) return BBGPU_ERR_CUDA;
    int rc = load_x(m, x, n);
    if (rc) return rc;
    cudaMemcpyAsync(m->t, t, sizeof(float) * n, cudaMemcpyHostToDevice, m->s);
    if (small_net(m)) {
        rows_pass(m, m->xf, m->t, n, 0, 0, 0);
        const SplitArgs S = wgrad_pass(m, n);
        k_split_sums<<<(unsigned)((m->np + 255) / 256), 256, 0, m->s>>>(m->np, S, m->g);
        k_sum<<<1, 256, 0, m->s>>>(n, m->r2, m->loss);
    } else {
        forward(m, n, m->t);
        backward(m, n);
    }
    float ls = 0.0f;
    if (grads) cudaMemcpyAsync(grads, m->g, sizeof(float) * m->np, cudaMemcpyDeviceToHost, m->s);
    cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->s);
    rc = finish(m);
    if (loss) *loss = ls / (float)n;
    return rc;
}

namespace {

// one Adam step on the n rows x, t, or step `step`'s minibatch of n rows of the set x, t of setn rows
void adam_step(bbgpu_mlp *m, const float *x, const float *t, int n, int setn, int step, uint64_t seed, float lr) {
    SplitArgs S{};
    if (small_net(m)) {
        rows_pass(m, x, t, n, setn, step, seed);
        S = wgrad_pass(m, n);
    } else {
        if (setn) k_gather_batch<<<n, 64, 0, m->s>>>(n, m->d, setn, seed, step, x, t, m->x16, m->t);
        forward(m, n, m->t);
        backward(m, n);
    }
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    k_adam<<<(unsigned)((m->np + 255) / 256), 256, 0, m->s>>>(m->np, m->w, m->m1, m->m2, m->g, S, m->w16, lr, b1, b2,
                                                              1.0f - powf(b1, (float)m->step),
                                                              1.0f - powf(b2, (float)m->step), 1e-8f);
}

// the sum of the squared residuals of the last step's n rows into m->loss
void step_loss(bbgpu_mlp *m, int n) {
    if (small_net(m)) k_sum<<<1, 256, 0, m->s>>>(n, m->r2, m->loss);
}

}  // namespace

extern "C" int bbgpu_mlp_train(bbgpu_mlp *m, const float *x, const float *t, long long n, int steps, int batch,
                               float lr, uint64_t seed, float *loss) {
    if (!m || !x || !t || n < 1 || n > 0x7fffffffLL || steps < 1 || batch < 1 || !(lr > 0)) return BBGPU_ERR_ARG;
    if (cudaSetDevice(m->device) != cudaSuccess) return BBGPU_ERR_CUDA;
    int rc = grow(m, batch);
    if (rc) return rc;
    if (n > m->set_cap) {
        cudaFree(m->set_x);
        cudaFree(m->set_t);
        m->set_x = m->set_t = nullptr;
        m->set_cap = 0;
        if (cudaMalloc(&m->set_x, sizeof(float) * (size_t)n * m->d) != cudaSuccess ||
            cudaMalloc(&m->set_t, sizeof(float) * (size_t)n) != cudaSuccess) {
            cudaGetLastError();
            return BBGPU_ERR_NOMEM;
        }
        m->set_cap = n;
    }
    cudaMemcpyAsync(m->set_x, x, sizeof(float) * (size_t)n * m->d, cudaMemcpyHostToDevice, m->s);
    cudaMemcpyAsync(m->set_t, t, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, m->s);
    for (int k = 0; k < steps; k++) adam_step(m, m->set_x, m->set_t, batch, (int)n, k, seed, lr);
    step_loss(m, batch);
    float ls = 0.0f;
    cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->s);
    rc = finish(m);
    if (loss) *loss = ls / (float)batch;
    return rc;
}

extern "C" int bbgpu_mlp_train_step(bbgpu_mlp *m, const float *x, const float *t, int n, float lr, float *loss) {
    if (!m || !x || !t || n < 1 || !(lr > 0)) return BBGPU_ERR_ARG;
    if (cudaSetDevice(m->device) != cudaSuccess) return BBGPU_ERR_CUDA;
    int rc = load_x(m, x, n);
    if (rc) return rc;
    cudaMemcpyAsync(m->t, t, sizeof(float) * n, cudaMemcpyHostToDevice, m->s);
    adam_step(m, m->xf, m->t, n, 0, 0, 0, lr);
    step_loss(m, n);
    float ls = 0.0f;
    cudaMemcpyAsync(&ls, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->s);
    rc = finish(m);
    if (loss) *loss = ls / (float)n;
    return rc;
}
