// Learned SDF surrogate: a Fourier-feature MLP trained on the GPU by this
// file's own kernels (forward, backward, Adam), with no library GEMM.
//
// Network (no counterpart in the reference; it stands in for an expensive
// many-primitive Source):
//   x (3, the source's world coordinates)
//   -> Fourier features, 16 frequencies per axis: sin(w_j x_a), cos(w_j x_a),
//      w_j = pi * 2^(7 j / 15), feature a*32 + 2j (+1 for cos)        96
//   -> 6 hidden layers of 256, softplus_beta(z) = log(1 + exp(beta z)) / beta
//      with beta = 100 (computed as max(z,0) + log1p(exp(-beta |z|)) / beta)
//   -> linear output (signed distance)                                  1
// Parameters (fp32 master copy, this order): W0[256][96], b0[256],
// W1..W5[256][256], b1..b5[256], w_out[256], b_out.
//
// Training data: points drawn uniformly in the domain box, kept with
// probability 1 near the surface (|f| < 0.05) and 0.25 elsewhere, labelled by
// the exact program (the same evaluator as the grid sampler).  Loss: L1
// against the target truncated to [-d, d] (one-sided where it saturates,
// see loss_l1), d = 0.1 by default.  Optimiser: Adam.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <utility>
#include <vector>

#include "internal.h"
#include "mlp.h"
#include "vm.cuh"

namespace iso {
namespace mlp {

// ---------------------------------------------------------------- helpers ---
__host__ __device__ __forceinline__ uint64_t splitmix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__host__ __device__ __forceinline__ float unit_float(uint64_t h) { return (float)(h >> 40) * (1.0f / 16777216.0f); }

__device__ __forceinline__ float softplus(float z) {
    return fmaxf(z, 0.0f) + log1pf(expf(-BETA * fabsf(z))) * (1.0f / BETA);
}
// d softplus_beta / dz = sigmoid(beta z)
__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-BETA * z)); }

__host__ __device__ __forceinline__ float freq(int j) { return 3.14159265358979f * exp2f((float)(7 * j) / 15.0f); }

// ------------------------------------------------------------ fp32 GEMM ---
// C[M x N] = A[M x K] * B[K x N] in fp32 FMAs, packed two rows to an
// instruction (fma.rn.f32x2: the FMA pipe's full rate from half of the issue
// slots, which leaves room for the shared-memory loads).  256 threads as 16 x
// 16, BM = 16 TM, BN = 16 TN, K steps of 8 by asynchronous copies, three steps
// ahead (through registers, ptxas sank the loads to where they were stored:
// 59 % of the FMA pipe, mostly waiting for them).
//   A_K: element (i, k) of A at A[i * lda + k], else at A[k * lda + i]
//   B_K: element (k, j) of B at B[j * ldb + k], else at B[k * ldb + j]
// M and K may be any numbers (M a multiple of 4 where A is not K-contiguous);
// N, lda and ldb are multiples of 4, the pointers are 16-byte
// aligned.
//   EPI_FORWARD   C = acc + bias[j] and C2 = softplus(C)
//   EPI_BACKWARD  C = acc * sigmoid(Z[i][j]), and colsum[tile row][j] = the tile's column sums
//   EPI_WEIGHTS   C += acc by atomics, K split over gridDim.z
// 65536 x 256 x 256 (8.6 GFLOP) on the GB300, whose FMA pipe reaches 77
// TFLOP/s: 0.17 ms as the weights' product (50 TFLOP/s, bound by the packed
// FMAs' register reads: 67 % of the pipe), 0.19 ms with either elementwise
// epilogue.  64 x 64 tiles with scalar loads and 4 x 4 per thread took 0.59
// and 0.67 ms, and 0.05-0.13 ms more for the elementwise passes, column sums
// and copies that the epilogues replace.  Scalar FMAs in the same tiles: 0.17
// and 0.21 ms.
enum Epilogue { EPI_FORWARD, EPI_BACKWARD, EPI_WEIGHTS };
constexpr int TK = 8;
constexpr int STAGES = 4;  // K steps of shared memory, three of them in flight

struct GemmArgs {
    int M, N, K;
    const float* A;
    const float* B;
    int lda, ldb;
    float* C;
    int ldc;
    const float* bias;  // EPI_FORWARD
    float* C2;          // EPI_FORWARD
    const float* Z;     // EPI_BACKWARD, laid out as C
    float* colsum;      // EPI_BACKWARD
};

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Asynchronous copy of one operand's tile, E rows (or columns) x TK, to
// s[k][e]; KC says whether k is its contiguous index (4 bytes at a time then,
// transposing; 16 otherwise).  Entries past the limits are zero.
template <int E, bool KC>
__device__ __forceinline__ void copy_tile(float (*s)[E + 4], const float* __restrict__ p, int ld, int e0, int elim,
                                          int k0, int klim) {
    if (KC) {
#pragma unroll
        for (int i = 0; i < E * TK / 256; ++i) {
            const int k = threadIdx.x % TK, e = threadIdx.x / TK + (256 / TK) * i;
            const bool in = e0 + e < elim && k0 + k < klim;
            const float* src = in ? p + (int64_t)(e0 + e) * ld + k0 + k : p;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(&s[k][e])),
                         "l"(src), "r"(in ? 4 : 0));
        }
    } else if (threadIdx.x < E * TK / 4) {
        const int k = threadIdx.x / (E / 4), e = 4 * (threadIdx.x % (E / 4));
        const bool in = e0 + e < elim && k0 + k < klim;
        const float* src = in ? p + (int64_t)(k0 + k) * ld + e0 + e : p;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&s[k][e])),
                     "l"(src), "r"(in ? 16 : 0));
    }
}

template <int TM, int TN, bool A_K, bool B_K, int EPI>
__global__ void __launch_bounds__(256, 2) gemm_f32(GemmArgs G) {
    constexpr int BM = 16 * TM, BN = 16 * TN;
    __shared__ __align__(16) float As[STAGES][TK][BM + 4];
    __shared__ __align__(16) float Bs[STAGES][TK][BN + 4];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int i0 = blockIdx.y * BM, j0 = blockIdx.x * BN;
    int kbeg = 0, kend = G.K;
    if (EPI == EPI_WEIGHTS) {
        const int per = ((G.K + (int)gridDim.z - 1) / (int)gridDim.z + TK - 1) / TK * TK;
        kbeg = min(G.K, (int)blockIdx.z * per);
        kend = min(G.K, kbeg + per);
    }
    uint64_t acc[TM / 2][TN] = {};  // pairs of rows
    const int steps = (kend - kbeg + TK - 1) / TK;
    auto fetch = [&](int step) {
        if (step < steps) {
            copy_tile<BM, A_K>(As[step % STAGES], G.A, G.lda, i0, G.M, kbeg + step * TK, kend);
            copy_tile<BN, B_K>(Bs[step % STAGES], G.B, G.ldb, j0, G.N, kbeg + step * TK, kend);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int step = 0; step < STAGES - 1; ++step) fetch(step);
    for (int step = 0; step < steps; ++step) {
        const int buf = step % STAGES;
        // this step's copies have landed, and every thread is done with the
        // step before, whose buffer the next copies take
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        fetch(step + STAGES - 1);
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            // rows ty*4.. (and BM/2 + ty*4..), columns tx*4.. (and BN/2 + tx*4..)
            uint64_t a[TM / 2], b[TN];
#pragma unroll
            for (int h = 0; h < TM / 4; ++h) {
                const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&As[buf][k][h * (BM / 2) + ty * 4]);
                a[2 * h] = q.x;
                a[2 * h + 1] = q.y;
            }
#pragma unroll
            for (int h = 0; h < TN / 4; ++h) {
                const float4 q = *reinterpret_cast<const float4*>(&Bs[buf][k][h * (BN / 2) + tx * 4]);
                b[4 * h] = pack2(q.x, q.x);
                b[4 * h + 1] = pack2(q.y, q.y);
                b[4 * h + 2] = pack2(q.z, q.z);
                b[4 * h + 3] = pack2(q.w, q.w);
            }
#pragma unroll
            for (int r = 0; r < TM / 2; ++r)
#pragma unroll
                for (int c = 0; c < TN; ++c) acc[r][c] = fma2(a[r], b[c], acc[r][c]);
        }
    }
    float col[TN] = {};
#pragma unroll
    for (int r = 0; r < TM; ++r) {
        const int gi = i0 + (r / 4) * (BM / 2) + ty * 4 + r % 4;
        if (gi >= G.M) continue;
#pragma unroll
        for (int h = 0; h < TN / 4; ++h) {
            const int gj = j0 + h * (BN / 2) + tx * 4;
            if (gj >= G.N) continue;
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 two = unpack2(acc[r / 2][4 * h + c]);
                v[c] = r % 2 ? two.y : two.x;
            }
            const int64_t at = (int64_t)gi * G.ldc + gj;
            if (EPI == EPI_FORWARD) {
                const float4 bb = __ldg(reinterpret_cast<const float4*>(G.bias + gj));
                const float4 z = make_float4(v[0] + bb.x, v[1] + bb.y, v[2] + bb.z, v[3] + bb.w);
                *reinterpret_cast<float4*>(G.C + at) = z;
                *reinterpret_cast<float4*>(G.C2 + at) =
                    make_float4(softplus(z.x), softplus(z.y), softplus(z.z), softplus(z.w));
            } else if (EPI == EPI_BACKWARD) {
                const float4 z = __ldg(reinterpret_cast<const float4*>(G.Z + at));
                const float4 d = make_float4(v[0] * sigmoid(z.x), v[1] * sigmoid(z.y), v[2] * sigmoid(z.z),
                                             v[3] * sigmoid(z.w));
                *reinterpret_cast<float4*>(G.C + at) = d;
                col[4 * h] += d.x;
                col[4 * h + 1] += d.y;
                col[4 * h + 2] += d.z;
                col[4 * h + 3] += d.w;
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) atomicAdd(G.C + at + c, v[c]);
            }
        }
    }
    if (EPI == EPI_BACKWARD) {
        // column sums of the tile: over the 16 thread rows in shared memory
        __syncthreads();  // the last step's tile is used
        float(*s_col)[BN] = reinterpret_cast<float(*)[BN]>(&Bs[0][0][0]);
#pragma unroll
        for (int c = 0; c < TN; ++c) s_col[ty][(c / 4) * (BN / 2) + tx * 4 + c % 4] = col[c];
        __syncthreads();
        for (int j = threadIdx.x; j < BN && j0 + j < G.N; j += 256) {
            float sum = 0.0f;
            for (int r = 0; r < 16; ++r) sum += s_col[r][j];
            G.colsum[(size_t)blockIdx.y * G.N + j0 + j] = sum;
        }
    }
}

// 128 x 128 tiles once they give every SM one (n x 256 outputs: n >= 64 per
// SM), else 64 x 64 ones, four times as many blocks.  (65536 x 256 outputs are
// 3.4 waves of two blocks to an SM; the last part of one as 64 x 128 tiles in
// a launch of its own took 164 + 40 us against 189: a block whose SM has
// fallen empty beside it already runs faster.)
// returns the number of tile rows
template <bool A_K, bool B_K, int EPI>
uint32_t gemm(cudaStream_t s, int sms, const GemmArgs& G) {
    if (EPI == EPI_WEIGHTS) {
        // K = the points: slices of at least 64, two blocks per SM
        const int tiles = ((G.N + 127) / 128) * ((G.M + 127) / 128);
        const int slices = std::max(1, std::min(2 * sms / tiles, (G.K + 63) / 64));
        gemm_f32<8, 8, A_K, B_K, EPI><<<dim3((G.N + 127) / 128, (G.M + 127) / 128, slices), 256, 0, s>>>(G);
        return (uint32_t)((G.M + 127) / 128);
    }
    if ((int64_t)((G.M + 127) / 128) * ((G.N + 127) / 128) < sms) {
        gemm_f32<4, 4, A_K, B_K, EPI><<<dim3((G.N + 63) / 64, (G.M + 63) / 64), 256, 0, s>>>(G);
        return (uint32_t)((G.M + 63) / 64);
    }
    gemm_f32<8, 8, A_K, B_K, EPI><<<dim3((G.N + 127) / 128, (G.M + 127) / 128), 256, 0, s>>>(G);
    return (uint32_t)((G.M + 127) / 128);
}

// ------------------------------------------------------- elementwise kernels ---
// one thread per frequency: its sine and cosine
__global__ void fourier(const float* pts, uint32_t n, float* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * (FF / 2)) return;
    const uint32_t p = i / (FF / 2), f = i % (FF / 2);
    const float x = freq(f % 16) * pts[3 * p + f / 16];
    float sn, cs;
    sincosf(x, &sn, &cs);
    reinterpret_cast<float2*>(out)[i] = make_float2(sn, cs);
}

// y[p] = a[p] . w + b; a warp for every four points, bound by the read of a
// (65536 points: 34 us with a point per warp and 4-byte loads)
__global__ void __launch_bounds__(256) out_forward(const float* __restrict__ a, uint32_t n, const float* __restrict__ w,
                                                   const float* b, float* __restrict__ y) {
    static_assert(HID == 256, "two float4 per lane");
    const uint32_t lane = threadIdx.x & 31, p0 = (blockIdx.x * 8 + threadIdx.x / 32) * 4;
    if (p0 >= n) return;
    const float4 w0 = __ldg(reinterpret_cast<const float4*>(w) + lane), w1 = __ldg(reinterpret_cast<const float4*>(w) + 32 + lane);
    float4 q[4][2];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const float4* row = reinterpret_cast<const float4*>(a + (size_t)min(p0 + j, n - 1) * HID);
        q[j][0] = __ldg(row + lane);
        q[j][1] = __ldg(row + 32 + lane);
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const float4 u = q[j][0], v = q[j][1];
        float s = ((u.x * w0.x + u.y * w0.y) + (u.z * w0.z + u.w * w0.w)) + ((v.x * w1.x + v.y * w1.y) + (v.z * w1.z + v.w * w1.w));
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        if (lane == 0 && p0 + j < n) y[p0 + j] = s + b[0];
    }
}

// Truncated L1: e = y - t inside the band |t| < d; where the target is
// saturated (t >= d or t <= -d) only a prediction on the band's side of +-d
// is penalised (e = min(y - d, 0) or max(y + d, 0)).  loss = mean |e|,
// dy = sign(e) / n; the loss accumulates into *loss and the sum of dy (the
// output bias' gradient) into *dsum.
__global__ void loss_l1(const float* y, const float* t, uint32_t n, float clampd, float* dy, float* loss,
                        float* dsum) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f, g = 0.0f;
    if (i < n) {
        const float ti = t[i], yi = y[i];
        const float d = (ti >= clampd) ? fminf(yi - clampd, 0.0f) : (ti <= -clampd) ? fmaxf(yi + clampd, 0.0f) : yi - ti;
        l = fabsf(d);
        g = (d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f)) / (float)n;
        dy[i] = g;
    }
    for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_xor_sync(0xFFFFFFFFu, l, o);
        g += __shfl_xor_sync(0xFFFFFFFFu, g, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(loss, l / (float)n);
        atomicAdd(dsum, g);
    }
}

// The backward pass of the output layer in one read of the last layer's z
// and a (a range of points per block; thread = four columns, every fourth
// point):
//   dz[p][k] = dy[p] w[k] sigmoid(z[p][k]), each block's column sums of it in
//   gb[block][k], and of dy[p] a[p][k] in gw[block][k]
// Bound by memory (65536 points: 200 MB; 86 us with a column per thread, whose
// 4-byte loads left too little in flight).
__global__ void __launch_bounds__(256) out_backward(const float* __restrict__ dy, const float* __restrict__ w,
                                                    const float* __restrict__ z, const float* __restrict__ a,
                                                    uint32_t n, float* __restrict__ dz, float* gw, float* gb) {
    static_assert(HID == 256, "64 threads cover a row");
    __shared__ float4 s_w[4][64], s_b[4][64];
    const uint32_t c = threadIdx.x % 64, g = threadIdx.x / 64;
    const uint32_t per = (n + gridDim.x - 1) / gridDim.x;
    const uint32_t p0 = blockIdx.x * per, p1 = min(n, p0 + per);
    const float4 wk = __ldg(reinterpret_cast<const float4*>(w) + c);
    float4 sw = make_float4(0.0f, 0.0f, 0.0f, 0.0f), sb = sw;
#pragma unroll 4
    for (uint32_t p = p0 + g; p < p1; p += 4) {
        const float d = __ldg(dy + p);
        const size_t at = (size_t)p * (HID / 4) + c;
        const float4 zz = __ldg(reinterpret_cast<const float4*>(z) + at), aa = __ldg(reinterpret_cast<const float4*>(a) + at);
        const float4 o = make_float4(d * wk.x * sigmoid(zz.x), d * wk.y * sigmoid(zz.y), d * wk.z * sigmoid(zz.z),
                                     d * wk.w * sigmoid(zz.w));
        reinterpret_cast<float4*>(dz)[at] = o;
        sb = make_float4(sb.x + o.x, sb.y + o.y, sb.z + o.z, sb.w + o.w);
        sw = make_float4(sw.x + d * aa.x, sw.y + d * aa.y, sw.z + d * aa.z, sw.w + d * aa.w);
    }
    s_w[g][c] = sw;
    s_b[g][c] = sb;
    __syncthreads();
    const float* fw = reinterpret_cast<const float*>(s_w);
    const float* fb = reinterpret_cast<const float*>(s_b);
    const uint32_t k = threadIdx.x;
    gw[(size_t)blockIdx.x * HID + k] = (fw[k] + fw[HID + k]) + (fw[2 * HID + k] + fw[3 * HID + k]);
    gb[(size_t)blockIdx.x * HID + k] = (fb[k] + fb[HID + k]) + (fb[2 * HID + k] + fb[3 * HID + k]);
}

// The gradients that are sums over the points (the biases', the output
// weights'), from the tiles' or blocks' partial sums: added in fp64, where
// hundreds of fp32 atomics on one word would each round the running sum.
struct ColumnSums {
    const float* part[NLAYERS + 1];  // rows x HID
    uint32_t rows[NLAYERS + 1];
    float* out[NLAYERS + 1];
};

__global__ void __launch_bounds__(1024) add_partials(ColumnSums S) {
    __shared__ double s_sum[32][32];
    const uint32_t c = threadIdx.x % 32, r0 = threadIdx.x / 32, k = 32 * blockIdx.x + c;
    const float* p = S.part[blockIdx.y] + k;
    double sum = 0.0;
#pragma unroll 8
    for (uint32_t r = r0; r < S.rows[blockIdx.y]; r += 32) sum += (double)__ldg(p + (size_t)r * HID);
    s_sum[r0][c] = sum;
    __syncthreads();
    if (r0) return;
    for (int w = 1; w < 32; ++w) sum += s_sum[w][c];
    S.out[blockIdx.y][k] = (float)sum;
}

__global__ void adam(float* p, const float* g, float* m, float* v, uint64_t n, float lr, float b1, float b2,
                     float eps, float c1, float c2) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// ------------------------------------------------------------- dataset ---
struct SampleArgs {
    ProgView pv;
    uint64_t seed;
    uint64_t base;     // candidate counter offset
    uint32_t ncand;
    float lo, hi;      // world box
    float near, far_keep;
    float* pts;        // world coordinates
    float* labels;
    uint32_t* count;
    uint32_t cap;
};

__global__ void make_samples(SampleArgs A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.ncand) return;
    const uint64_t id = A.base + i;
    const float x = A.lo + (A.hi - A.lo) * unit_float(splitmix(A.seed ^ (3 * id)));
    const float y = A.lo + (A.hi - A.lo) * unit_float(splitmix(A.seed ^ (3 * id + 1)));
    const float z = A.lo + (A.hi - A.lo) * unit_float(splitmix(A.seed ^ (3 * id + 2)));
    const float f = eval_scalar(A.pv, v3(x, y, z));
    const float u = unit_float(splitmix(A.seed * 31 + id));
    if (!(fabsf(f) < A.near || u < A.far_keep)) return;
    const uint32_t at = atomicAdd(A.count, 1u);
    if (at >= A.cap) return;
    A.pts[3 * at] = x;
    A.pts[3 * at + 1] = y;
    A.pts[3 * at + 2] = z;
    A.labels[at] = f;
}

__global__ void gather_batch(const float* pts, const float* labels, uint32_t n, uint64_t seed, uint32_t b,
                             float* bp, float* bl) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b) return;
    const uint32_t k = (uint32_t)(splitmix(seed + i) % n);
    bp[3 * i] = pts[3 * k];
    bp[3 * i + 1] = pts[3 * k + 1];
    bp[3 * i + 2] = pts[3 * k + 2];
    bl[i] = labels[k];
}

}  // namespace mlp
}  // namespace iso

using namespace iso;
using namespace iso::mlp;


namespace {

struct Views {
    float *pts, *ff, *z[NLAYERS], *a[NLAYERS], *y, *t, *dy, *d[2], *part, *loss;
    uint32_t part_rows;  // rows of each of part's NLAYERS + 1 arrays
};

// partial sums per column: a row per 64 points (the smaller GEMM tile) or per block of out_backward
inline uint32_t partial_rows(const iso_mlp* net, uint32_t n) { return std::max<uint32_t>((n + 63) / 64, 4 * (uint32_t)net->ctx->sms); }

// each piece starts on a 256-byte boundary (the GEMMs load 16 bytes at once)
inline size_t piece(size_t floats) { return (floats + 63) & ~(size_t)63; }

iso_status ensure_work(iso_mlp* net, uint32_t n) {
    if (n <= net->cap && net->work) return ISO_OK;
    if (net->work) cudaFree(net->work);
    net->work = nullptr;
    const size_t floats = piece(3 * (size_t)n) + piece(FF * (size_t)n) + (2 * NLAYERS + 2) * piece(HID * (size_t)n) +
                          3 * piece(n) + (NLAYERS + 1) * piece(HID * (size_t)partial_rows(net, n)) + 1024;
    cudaError_t e = cudaMalloc(&net->work, floats * 4);
    if (e != cudaSuccess) return cuda_fail(net->ctx, e, "mlp work");
    net->work_bytes = floats * 4;
    net->cap = n;
    return ISO_OK;
}

Views views(iso_mlp* net) {
    Views w;
    float* p = net->work;
    const size_t n = net->cap;
    auto take = [&](size_t floats) {
        float* at = p;
        p += piece(floats);
        return at;
    };
    w.pts = take(3 * n);
    w.ff = take(FF * n);
    for (int l = 0; l < NLAYERS; ++l) w.z[l] = take(HID * n);
    for (int l = 0; l < NLAYERS; ++l) w.a[l] = take(HID * n);
    w.y = take(n);
    w.t = take(n);
    w.dy = take(n);
    w.d[0] = take(HID * n);
    w.d[1] = take(HID * n);
    w.part_rows = partial_rows(net, net->cap);
    w.part = take((NLAYERS + 1) * (size_t)HID * w.part_rows);
    w.loss = p;
    return w;
}

inline unsigned blocks(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// forward over w.pts[0..n) into w.y; keeps z/a for backward
void forward(iso_mlp* net, const Views& w, uint32_t n) {
    cudaStream_t s = net->ctx->stream;
    const float* P = net->params;
    fourier<<<blocks((uint64_t)n * (FF / 2), 256), 256, 0, s>>>(w.pts, n, w.ff);
    for (int l = 0; l < NLAYERS; ++l) {
        // z = in [n x in_dim] * W^T [in_dim x HID] + b, a = softplus(z)
        const int in_dim = l ? HID : FF;
        GemmArgs g{(int)n, HID, in_dim, l ? w.a[l - 1] : w.ff, P + weight_offset(l), in_dim, in_dim, w.z[l], HID};
        g.bias = P + bias_offset(l);
        g.C2 = w.a[l];
        gemm<true, true, EPI_FORWARD>(s, net->ctx->sms, g);
    }
    out_forward<<<blocks(n, 32), 256, 0, s>>>(w.a[NLAYERS - 1], n, P + OUT_W, P + OUT_B, w.y);
    net->ctx->launches += 2 + NLAYERS;
}

// grads (zeroed first) of the loss over n points with targets w.t; *loss
void backward(iso_mlp* net, const Views& w, uint32_t n, float clampd) {
    cudaStream_t s = net->ctx->stream;
    const float* P = net->params;
    float* G = net->grads;
    cudaMemsetAsync(G, 0, NPARAMS * 4, s);
    cudaMemsetAsync(w.loss, 0, 4, s);
    loss_l1<<<blocks(n, 256), 256, 0, s>>>(w.y, w.t, n, clampd, w.dy, w.loss, G + OUT_B);
    // dz of the last layer and the output layer's gradients
    const int last = NLAYERS - 1;
    float *dz = w.d[0], *below = w.d[1];
    ColumnSums sums{};  // entry l: layer l's biases; the last: the output weights
    for (int l = 0; l <= NLAYERS; ++l) {
        sums.part[l] = w.part + (size_t)l * HID * w.part_rows;
        sums.out[l] = G + (l < NLAYERS ? bias_offset(l) : OUT_W);
    }
    const unsigned out_blocks = std::min<unsigned>(blocks(n, 16), 4 * (unsigned)net->ctx->sms);
    sums.rows[last] = sums.rows[NLAYERS] = out_blocks;
    out_backward<<<out_blocks, 256, 0, s>>>(w.dy, P + OUT_W, w.z[last], w.a[last], n, dz,
                                            const_cast<float*>(sums.part[NLAYERS]), const_cast<float*>(sums.part[last]));
    for (int l = last; l >= 0; --l) {
        const int in_dim = l ? HID : FF;
        // dW = dz^T [HID x n] * in [n x in_dim]
        gemm<false, false, EPI_WEIGHTS>(s, net->ctx->sms,
                                        GemmArgs{HID, in_dim, (int)n, dz, l ? w.a[l - 1] : w.ff, HID, in_dim,
                                                 G + weight_offset(l), in_dim});
        if (l > 0) {
            // dz of the layer below = (dz [n x HID] * W [HID x HID]) sigmoid(z), and its bias' gradient
            GemmArgs g{(int)n, HID, HID, dz, P + weight_offset(l), HID, HID, below, HID};
            g.Z = w.z[l - 1];
            g.colsum = const_cast<float*>(sums.part[l - 1]);
            sums.rows[l - 1] = gemm<true, false, EPI_BACKWARD>(s, net->ctx->sms, g);
            std::swap(dz, below);
        }
    }
    add_partials<<<dim3(HID / 32, NLAYERS + 1), 1024, 0, s>>>(sums);
    net->ctx->launches += 2 + 2 * NLAYERS;
}

}  // namespace

extern "C" {

iso_status iso_mlp_create(iso_ctx* ctx, uint64_t seed, iso_mlp** out) {
    if (!ctx || !out) return ISO_ERR_INVALID_ARG;
    *out = nullptr;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    iso_mlp* net = new iso_mlp();
    net->ctx = ctx;
    cudaError_t e = cudaMalloc(&net->params, 4ull * NPARAMS * 4);
    if (e != cudaSuccess) {
        delete net;
        return cuda_fail(ctx, e, "mlp params");
    }
    net->grads = net->params + NPARAMS;
    net->m = net->grads + NPARAMS;
    net->v = net->m + NPARAMS;
    // uniform(-a, a) with a = sqrt(6 / (fan_in + fan_out)); biases zero
    std::vector<float> h(NPARAMS, 0.0f);
    for (int l = 0; l <= NLAYERS; ++l) {
        const int fin = l == 0 ? FF : HID, fout = l == NLAYERS ? 1 : HID;
        const float a = std::sqrt(6.0f / (float)(fin + fout));
        const size_t off = l == NLAYERS ? OUT_W : weight_offset(l);
        for (size_t k = 0; k < (size_t)fin * fout; ++k)
            h[off + k] = a * (2.0f * unit_float(splitmix(seed * 1000003ull + off + k)) - 1.0f);
    }
    e = upload(ctx, net->params, h.data(), 4ull * NPARAMS);
    if (e == cudaSuccess) e = cudaMemsetAsync(net->m, 0, 8ull * NPARAMS, ctx->stream);
    if (e != cudaSuccess) {
        iso_mlp_destroy(net);
        return cuda_fail(ctx, e, "mlp init");
    }
    mlp_infer_invalidate(net, h.data());
    *out = net;
    return ISO_OK;
}

iso_status iso_mlp_destroy(iso_mlp* net) {
    if (!net) return ISO_ERR_INVALID_ARG;
    cudaSetDevice(net->ctx->device);
    if (net->params) cudaFree(net->params);
    if (net->work) cudaFree(net->work);
    if (net->data_pts) cudaFree(net->data_pts);
    mlp_infer_release(net);
    delete net;
    return ISO_OK;
}

uint64_t iso_mlp_num_params(void) { return NPARAMS; }

iso_status iso_mlp_get_params(iso_mlp* net, float* host) {
    if (!net || !host) return ISO_ERR_INVALID_ARG;
    cudaError_t e = download(net->ctx, host, net->params, 4ull * NPARAMS);
    return e == cudaSuccess ? ISO_OK : cuda_fail(net->ctx, e, "get params");
}

iso_status iso_mlp_set_params(iso_mlp* net, const float* host) {
    if (!net || !host) return ISO_ERR_INVALID_ARG;
    cudaError_t e = upload(net->ctx, net->params, host, 4ull * NPARAMS);
    if (e == cudaSuccess) e = cudaStreamSynchronize(net->ctx->stream);  // the caller's memory may be page-locked
    mlp_infer_invalidate(net, e == cudaSuccess ? host : nullptr);
    return e == cudaSuccess ? ISO_OK : cuda_fail(net->ctx, e, "set params");
}

// fp32 forward of n host points (world coordinates) into host values
iso_status iso_mlp_forward(iso_mlp* net, const float* pts, uint32_t n, float* values) {
    if (!net || (!pts && n) || (!values && n)) return ISO_ERR_INVALID_ARG;
    if (n == 0) return ISO_OK;
    iso_status s = set_device(net->ctx);
    if (s != ISO_OK || (s = ensure_work(net, n)) != ISO_OK) return s;
    Views w = views(net);
    cudaStream_t st = net->ctx->stream;
    cudaMemcpyAsync(w.pts, pts, 12ull * n, cudaMemcpyHostToDevice, st);
    {
        StageTimer timer(net->ctx, ISO_STAGE_MLP);
        forward(net, w, n);
    }
    cudaMemcpyAsync(values, w.y, 4ull * n, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? check_launch(net->ctx, "mlp forward") : cuda_fail(net->ctx, e, "mlp forward");
}

// loss and gradient of the training loss over given points/targets (host)
iso_status iso_mlp_loss_grad(iso_mlp* net, const float* pts, const float* targets, uint32_t n, float clampd,
                             float* loss, float* grad_host) {
    if (!net || !pts || !targets || n == 0) return ISO_ERR_INVALID_ARG;
    iso_status s = set_device(net->ctx);
    if (s != ISO_OK || (s = ensure_work(net, n)) != ISO_OK) return s;
    Views w = views(net);
    cudaStream_t st = net->ctx->stream;
    cudaMemcpyAsync(w.pts, pts, 12ull * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(w.t, targets, 4ull * n, cudaMemcpyHostToDevice, st);
    forward(net, w, n);
    backward(net, w, n, clampd);
    if (loss) cudaMemcpyAsync(loss, w.loss, 4, cudaMemcpyDeviceToHost, st);
    if (grad_host) cudaMemcpyAsync(grad_host, net->grads, 4ull * NPARAMS, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? check_launch(net->ctx, "mlp loss/grad") : cuda_fail(net->ctx, e, "mlp loss/grad");
}

// draw n samples in [lo, hi]^3 labelled by `exact` (see file comment)
iso_status iso_mlp_make_dataset(iso_mlp* net, const iso_program* exact, uint32_t n, float lo, float hi,
                                uint64_t seed) {
    iso::NvtxRange nvtx_range("iso_mlp_make_dataset");
    if (!net || !exact || n == 0) return ISO_ERR_INVALID_ARG;
    iso_status s = set_device(net->ctx);
    if (s != ISO_OK) return s;
    if (net->data_pts) cudaFree(net->data_pts);
    net->data_pts = nullptr;
    cudaError_t e = cudaMalloc(&net->data_pts, 16ull * n + 256);
    if (e != cudaSuccess) return cuda_fail(net->ctx, e, "dataset");
    net->data_labels = net->data_pts + 3ull * n;
    uint32_t* count = (uint32_t*)(net->data_labels + n);
    cudaStream_t st = net->ctx->stream;
    cudaMemsetAsync(count, 0, 4, st);
    uint64_t base = 0;
    uint32_t have = 0;
    for (int round = 0; round < 64 && have < n; ++round) {
        const uint32_t cand = std::max<uint32_t>(n, 1u << 20);
        SampleArgs a{exact->view(), seed, base, cand, lo, hi, 0.05f, 0.25f, net->data_pts, net->data_labels, count, n};
        {
            StageTimer timer(net->ctx, ISO_STAGE_MLP);
            make_samples<<<blocks(cand, 128), 128, 0, st>>>(a);
        }
        net->ctx->launches++;
        base += cand;
        e = cudaMemcpyAsync(&have, count, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_fail(net->ctx, e, "dataset");
    }
    net->data_n = std::min(have, n);
    return net->data_n == n ? ISO_OK : fail(net->ctx, ISO_ERR_CAPACITY, "dataset rounds exhausted");
}

// steps of Adam on random batches of the dataset; loss per step into history (nullable)
iso_status iso_mlp_train(iso_mlp* net, uint32_t steps, uint32_t batch, float lr, float clampd, uint64_t seed,
                         float* history) {
    iso::NvtxRange nvtx_range("iso_mlp_train");
    if (!net || batch == 0 || net->data_n == 0) return ISO_ERR_INVALID_ARG;
    iso_status s = set_device(net->ctx);
    if (s != ISO_OK || (s = ensure_work(net, batch)) != ISO_OK) return s;
    Views w = views(net);
    cudaStream_t st = net->ctx->stream;
    std::vector<float> hist(steps, 0.0f);
    float* d_hist = nullptr;
    if (history) {
        cudaError_t e = cudaMalloc(&d_hist, 4ull * std::max<uint32_t>(steps, 1));
        if (e != cudaSuccess) return cuda_fail(net->ctx, e, "history");
    }
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (uint32_t k = 0; k < steps; ++k) {
        StageTimer timer(net->ctx, ISO_STAGE_MLP);
        gather_batch<<<blocks(batch, 256), 256, 0, st>>>(net->data_pts, net->data_labels, net->data_n,
                                                          splitmix(seed + 7919ull * (net->step + 1)), batch, w.pts, w.t);
        forward(net, w, batch);
        backward(net, w, batch, clampd);
        ++net->step;
        const float c1 = 1.0f - std::pow(b1, (float)net->step), c2 = 1.0f - std::pow(b2, (float)net->step);
        // cosine decay to 5% of lr over the call
        const float lr_k = lr * (0.05f + 0.95f * 0.5f * (1.0f + std::cos(3.14159265f * (float)k / (float)steps)));
        adam<<<blocks(NPARAMS, 256), 256, 0, st>>>(net->params, net->grads, net->m, net->v, NPARAMS, lr_k, b1, b2,
                                                    eps, c1, c2);
        if (d_hist) cudaMemcpyAsync(d_hist + k, w.loss, 4, cudaMemcpyDeviceToDevice, st);
        net->ctx->launches += 2;
    }
    mlp_infer_invalidate(net);
    cudaError_t e = cudaSuccess;
    if (d_hist) {
        e = cudaMemcpyAsync(history, d_hist, 4ull * steps, cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (d_hist) cudaFree(d_hist);
    return e == cudaSuccess ? check_launch(net->ctx, "mlp train") : cuda_fail(net->ctx, e, "mlp train");
}

// ------------------------------------------------------------- checkpoints ---
// 32-byte header, then NPARAMS fp32 parameters, Adam's first and second
// moments; host byte order (little-endian on both supported machines).
namespace {
constexpr char CKPT_MAGIC[8] = {'I', 'S', 'O', 'M', 'L', 'P', '0', '1'};
struct CkptHeader {
    char magic[8];
    uint32_t version;       // 1
    uint32_t header_bytes;  // 32
    uint64_t nparams;
    uint64_t step;          // Adam steps taken
};
static_assert(sizeof(CkptHeader) == 32, "checkpoint header layout");

// 0 = ok, 1 = cannot open / short file, 2 = not a checkpoint of this network
int read_header(FILE* f, CkptHeader* h) {
    if (std::fread(h, sizeof(*h), 1, f) != 1) return 1;
    if (std::memcmp(h->magic, CKPT_MAGIC, 8) != 0 || h->version != 1 || h->header_bytes != sizeof(*h) ||
        h->nparams != NPARAMS)
        return 2;
    return 0;
}
}  // namespace

iso_status iso_mlp_checkpoint_info(const char* path, uint64_t* nparams, uint64_t* step) {
    if (!path) return ISO_ERR_INVALID_ARG;
    FILE* f = std::fopen(path, "rb");
    if (!f) return ISO_ERR_INVALID_ARG;
    CkptHeader h;
    const int r = read_header(f, &h);
    std::fseek(f, 0, SEEK_END);
    const long size = std::ftell(f);
    std::fclose(f);
    if (r != 0 || size != (long)(sizeof(h) + 12ull * NPARAMS)) return ISO_ERR_INVALID_ARG;
    if (nparams) *nparams = h.nparams;
    if (step) *step = h.step;
    return ISO_OK;
}

iso_status iso_mlp_save(iso_mlp* net, const char* path) {
    if (!net || !path) return ISO_ERR_INVALID_ARG;
    iso_status s = set_device(net->ctx);
    if (s != ISO_OK) return s;
    std::vector<float> host(3 * NPARAMS);
    cudaError_t e = download(net->ctx, host.data(), net->params, 4ull * NPARAMS);
    if (e == cudaSuccess) e = download(net->ctx, host.data() + NPARAMS, net->m, 8ull * NPARAMS);
    if (e != cudaSuccess) return cuda_fail(net->ctx, e, "checkpoint read");
    CkptHeader h{};
    std::memcpy(h.magic, CKPT_MAGIC, 8);
    h.version = 1;
    h.header_bytes = sizeof(h);
    h.nparams = NPARAMS;
    h.step = net->step;
    FILE* f = std::fopen(path, "wb");
    if (!f) return fail(net->ctx, ISO_ERR_INVALID_ARG, std::string("cannot write ") + path);
    const bool ok = std::fwrite(&h, sizeof(h), 1, f) == 1 &&
                    std::fwrite(host.data(), 4, host.size(), f) == host.size();
    if (std::fclose(f) != 0 || !ok) return fail(net->ctx, ISO_ERR_INVALID_ARG, std::string("cannot write ") + path);
    return ISO_OK;
}

iso_status iso_mlp_load(iso_mlp* net, const char* path) {
    if (!net || !path) return ISO_ERR_INVALID_ARG;
    iso_status s = iso_mlp_checkpoint_info(path, nullptr, nullptr);
    if (s != ISO_OK) return fail(net->ctx, s, std::string("not a checkpoint of this network: ") + path);
    if ((s = set_device(net->ctx)) != ISO_OK) return s;
    FILE* f = std::fopen(path, "rb");
    if (!f) return fail(net->ctx, ISO_ERR_INVALID_ARG, std::string("cannot read ") + path);
    CkptHeader h;
    std::vector<float> host(3 * NPARAMS);
    const bool ok = read_header(f, &h) == 0 && std::fread(host.data(), 4, host.size(), f) == host.size();
    std::fclose(f);
    if (!ok) return fail(net->ctx, ISO_ERR_INVALID_ARG, std::string("cannot read ") + path);
    // parameters | gradients | first moments | second moments, one allocation
    cudaError_t e = upload(net->ctx, net->params, host.data(), 4ull * NPARAMS);
    if (e == cudaSuccess) e = upload(net->ctx, net->m, host.data() + NPARAMS, 8ull * NPARAMS);
    if (e != cudaSuccess) return cuda_fail(net->ctx, e, "checkpoint load");
    net->step = h.step;
    mlp_infer_invalidate(net, host.data());
    return ISO_OK;
}

}  // extern "C"
