// BF16 tensor-core inference of the surrogate MLP on sm_103a (tcgen05).
//
// One CTA per SM runs two tiles of M = 128 points at a time through the whole
// network, so that one tile's matrix products run on the tensor cores while
// the other's activations run on the SM's own pipes:
//   * features / activations: the A operand of each tile, 128 rows x K bf16 in
//     shared memory, K-major with the 128-byte swizzle, as K-blocks of 64
//     columns (16 KB each; layer 0's 96 features are padded to 128);
//   * weights: the B operand, 256 rows (N) x 64 K bf16 per K-block (32 KB),
//     the same layout, copied by TMA bulk copies from a pre-swizzled bf16
//     image made once per parameter update (prepare_images) through a ring of
//     three slots by a producer thread that runs ahead;
//   * one thread issues tcgen05.mma.cta_group::1.kind::f16 (M=128, N=256,
//     K=16, fp32 accumulate) for the two tiles' layers in turn, each into its
//     own 256 TMEM columns, and commits to an mbarrier; every wait is bounded
//     (error flag, copies drained, TMEM freed);
//   * epilogue: eight warps per tile read the accumulator with tcgen05.ld (warp
//     w: 32 lanes = rows, 128 columns), add the bias, apply softplus_beta and
//     write the bf16 operand of the next layer; after the last layer they dot
//     with w_out (fp32) instead, and make the next tile's features.
// What bounds it is the SM's shared-memory / L1 bandwidth: a tile's layer
// moves 192 KB of MMA operands, 128 KB of weights in and 64 KB of activations
// out (3072 cycles at 128 bytes, against 2048 of MMA).  250001 points: 0.293
// ms with one tile at a time (products and activations in turn), 0.219 with
// two, 0.197 with the biases by value (read from memory they took another
// 128 KB per tile and layer).  Pairs of CTAs sharing the weights by multicast
// copies changed nothing.
// Descriptor formats (tcgen05 shared-memory matrix descriptor and the
// kind::f16 instruction descriptor) follow the PTX ISA for sm_100-class MMA.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "internal.h"
#include "mlp.h"

using namespace iso;
using namespace iso::mlp;

struct MlpImages {
    __nv_bfloat16* w = nullptr;  // per layer: NK/64 K-blocks of 256 rows x 128 B, swizzled
    float* bias = nullptr;       // NLAYERS x 256
    float* wout = nullptr;       // 256 + 1
    std::vector<float> host;     // bias, then wout: the kernel takes them by value
    bool host_valid = false;
    bool valid = false;
};

namespace {

constexpr int KB0 = 2;                 // layer 0: K padded 96 -> 128
constexpr int KB = HID / 64;           // layers 1..5: K = 256
constexpr size_t KBLOCK_BYTES_B = 256 * 128;   // 256 rows x 64 bf16
constexpr size_t KBLOCK_BYTES_A = 128 * 128;   // 128 rows x 64 bf16
constexpr uint32_t WAIT_LIMIT = 1u << 26;
constexpr uint64_t WAIT_NS = 1000000000ull;  // 1 s

__host__ __device__ constexpr size_t image_offset(int l) {  // in bf16 elements
    return l == 0 ? 0 : (size_t)KB0 * 256 * 64 + (size_t)(l - 1) * KB * 256 * 64;
}
constexpr size_t IMAGE_ELEMS = image_offset(NLAYERS);

// byte offset of element (row, k) in a swizzled K-major operand of `rows` rows
__host__ __device__ __forceinline__ uint32_t swz(uint32_t row, uint32_t k, uint32_t rows) {
    const uint32_t kb = k >> 6, c = (k & 63) >> 3, e = k & 7;
    return kb * rows * 128 + row * 128 + ((c ^ (row & 7)) << 4) + e * 2;
}

__global__ void prepare_images(const float* params, __nv_bfloat16* w, float* bias, float* wout) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    // weights
    if (i < IMAGE_ELEMS) {
        int l = 0;
        while (l + 1 < NLAYERS && i >= image_offset(l + 1)) ++l;
        const uint32_t local = i - (uint32_t)image_offset(l);
        const uint32_t K = l == 0 ? FF : HID;
        const uint32_t row = local / (l == 0 ? KB0 * 64 : KB * 64), k = local % (l == 0 ? KB0 * 64 : KB * 64);
        const float v = k < K ? params[weight_offset(l) + (size_t)row * K + k] : 0.0f;
        unsigned char* base = reinterpret_cast<unsigned char*>(w + image_offset(l));
        *reinterpret_cast<__nv_bfloat16*>(base + swz(row, k, 256)) = __float2bfloat16_rn(v);
    }
    if (i < NLAYERS * HID) bias[i] = params[bias_offset(i / HID) + i % HID];
    if (i < HID + 1) wout[i] = params[OUT_W + i];
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);  // start address
    d |= (uint64_t)1 << 16;                   // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                   // descriptor version
    d |= (uint64_t)2 << 61;                   // 128-byte swizzle
    return d;
}

// kind::f16: fp32 D, bf16 A and B, both K-major, N = 256, M = 128
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(IDESC), "r"(acc));
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// parity wait on an mbarrier, bounded in polls and in time (about a second);
// also given up once another role of the CTA gave up (*abort)
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t phase, const volatile uint32_t* abort) {
    uint64_t t0 = 0;
    for (uint32_t it = 0; it < WAIT_LIMIT; ++it) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(phase)
            : "memory");
        if (done) return true;
        if ((it & 63u) == 63u) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > WAIT_NS || (abort && *abort)) return false;
        }
    }
    return false;
}

// 32 lanes x 16 columns of 32 bits from TMEM, without waiting
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// wait for this thread's TMEM loads; the registers are tied to the wait so
// that no use of them moves above it
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}

// packed f32x2 arithmetic (two lanes per instruction on sm_100-class SMs)
__device__ __forceinline__ uint64_t f2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void uf2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// softplus_beta of z + b for two lanes at once:
//   max(x, 0) + log1p(u) / beta,  u = exp(-beta |x|) = 2^(-|x| beta log2(e)),
// u from the MUFU, log1p(u) / beta = u * P(u) with P a degree-4 polynomial
// fitted here to log1p(u) / (beta u) on [0, 1] (least squares at Chebyshev
// nodes; maximum absolute error 1e-7 after the 1/beta scaling, far below the
// bf16 rounding of the result)
__device__ __forceinline__ uint64_t softplus2(uint64_t z, uint64_t b) {
    constexpr float K = BETA * 1.4426950408889634f;
    const uint64_t x = add2(z, b);
    float t0, t1;
    uf2(mul2(x, f2(K, K)), t0, t1);
    const uint64_t u = f2(ex2_approx(-fabsf(t0)), ex2_approx(-fabsf(t1)));
    uint64_t p = fma2(f2(0.000321511645f, 0.000321511645f), u, f2(-0.00136042002f, -0.00136042002f));
    p = fma2(p, u, f2(0.00289453869f, 0.00289453869f));
    p = fma2(p, u, f2(-0.00491900276f, -0.00491900276f));
    p = fma2(p, u, f2(0.00999494363f, 0.00999494363f));
    float x0, x1;
    uf2(x, x0, x1);
    return fma2(u, p, f2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f)));
}


__device__ __forceinline__ float ffreq(int j) { return 3.14159265358979f * exp2f((float)(7 * j) / 15.0f); }

// sin and cos of a = w_j x (|a| < ~500): Cody-Waite reduction by 2 pi with a
// two-term constant (the high term has 8 significant bits, so n * hi is exact
// for |n| < 2^16), then the MUFU sine / cosine on [-pi, pi]
__device__ __forceinline__ void sincos_reduced(float a, float* s, float* c) {
    constexpr float TWO_PI_HI = 6.28125f;
    constexpr float TWO_PI_LO = 1.9353071795864769e-3f;
    const float n = rintf(a * 0.15915494309189535f);
    float r = fmaf(-n, TWO_PI_HI, a);
    r = fmaf(-n, TWO_PI_LO, r);
    __sincosf(r, s, c);
}

struct InferArgs {
    const unsigned char* w;  // swizzled bf16 weight image (K-blocks of 32 KB)
    // by value, so that the epilogue reads them through the constant cache:
    // loaded from memory, each lane's copy of 128 biases per layer took a
    // quarter of the shared-memory / L1 bandwidth, which bounds this kernel
    float bias[NLAYERS * HID];
    float wout[HID + 4];
    // points: either explicit (pts != null, n points, out[i]) or a grid of
    // nx x ny x nz lattice points (i, j, k) at p = (i*step*inv, j*step*inv,
    // k*step*inv) mapped by q = p * scale + offset, out[(k*ny + j)*nx + i]
    const float* pts;
    uint64_t n;
    uint32_t nx, ny, nz, step;
    float inv;
    float scale[3], offset[3];
    uint32_t groups;  // tiles a CTA works on at a time: 1 or 2
    float* out;
    uint32_t* err;
};

__device__ __forceinline__ void point_of(const InferArgs& A, uint64_t i, float* q) {
    if (A.pts) {
        q[0] = A.pts[3 * i];
        q[1] = A.pts[3 * i + 1];
        q[2] = A.pts[3 * i + 2];
        return;
    }
    const uint32_t x = (uint32_t)(i % A.nx);
    const uint64_t r = i / A.nx;
    const uint32_t y = (uint32_t)(r % A.ny), z = (uint32_t)(r / A.ny);
    // unfused, so that a host computing the same points in f32 feeds the
    // network identical coordinates
    q[0] = __fadd_rn(__fmul_rn(__fmul_rn((float)(x * A.step), A.inv), A.scale[0]), A.offset[0]);
    q[1] = __fadd_rn(__fmul_rn(__fmul_rn((float)(y * A.step), A.inv), A.scale[1]), A.offset[1]);
    q[2] = __fadd_rn(__fmul_rn(__fmul_rn((float)(z * A.step), A.inv), A.scale[2]), A.offset[2]);
}

constexpr int GROUP = 256;                 // threads of a tile's epilogue
constexpr int THREADS = 2 * GROUP + 64;    // two tiles, the MMA warp, the copying warp
constexpr int SLOTS = 3;                   // weight K-blocks in flight
constexpr size_t SMEM_A = 4 * KBLOCK_BYTES_A;                   // 64 KB: one tile's activations, 4 K-blocks
constexpr size_t SMEM_B = SLOTS * KBLOCK_BYTES_B;               // 96 KB: weight slots
constexpr size_t SMEM_TOTAL = 2 * SMEM_A + SMEM_B + 1024;       // + alignment slack

__host__ __device__ constexpr int kblocks_of(int l) { return l == 0 ? KB0 : KB; }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void commit_to(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

// a barrier of the 256 threads of group g; whether `ok` held for all of them
__device__ __forceinline__ bool group_all(int g, bool ok) {
    uint32_t all;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.and.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(all)
        : "r"((uint32_t)ok), "r"(1 + g), "r"(GROUP)
        : "memory");
    return all != 0;
}

// Fourier features of point q as row `row` of a tile's operand: k in
// [64*half, 64*half + 64) (96..127 zero)
__device__ __forceinline__ void write_features(unsigned char* sA, int row, int half, const float* q) {
    for (int k0 = 64 * half; k0 < 64 * half + 64; k0 += 8) {
        uint32_t packed[4] = {0u, 0u, 0u, 0u};
        if (k0 < FF) {
            const int a = k0 / 32;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = (k0 % 32) / 2 + i;
                float s, c;
                sincos_reduced(ffreq(j) * q[a], &s, &c);
                __nv_bfloat162 h = __floats2bfloat162_rn(s, c);
                packed[i] = *reinterpret_cast<uint32_t*>(&h);
            }
        }
        *reinterpret_cast<uint4*>(sA + swz(row, k0, 128)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
}

// Barriers (per tile g: ready = its operand is written, one arrival per warp; acc =
// its layer's MMAs are done; per slot: full = the K-block has landed, empty =
// the MMAs that read it are done).  Tile g's chain is ready -> MMA -> acc ->
// epilogue -> ready ...; the MMA thread takes the chains' steps in turn, so
// while it works on one tile the other's epilogue runs.  The operand and the
// accumulator need no second copy: the epilogue writes and reads them after
// acc (the MMAs are done with both), the MMAs after ready.
// Every wait is bounded; a role that gives up raises s_abort, which ends the
// others' waits; the MMAs and copies in flight are then waited for (again
// with a limit) before TMEM is freed.
__global__ void __launch_bounds__(THREADS, 1) mlp_infer_kernel(const __grid_constant__ InferArgs A) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t s_full[SLOTS], s_empty[SLOTS], s_ready[2], s_acc[2], s_drain;
    __shared__ uint32_t s_tmem;
    __shared__ volatile uint32_t s_abort;
    __shared__ float s_part[2][128];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sB = smem_u32(smem + 2 * SMEM_A);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full0 = smem_u32(&s_full[0]), empty0 = smem_u32(&s_empty[0]);
    const uint32_t ready0 = smem_u32(&s_ready[0]), acc0 = smem_u32(&s_acc[0]), drain = smem_u32(&s_drain);
    const uint64_t ntiles = (A.n + 127) / 128;
    const uint64_t steps = (ntiles + A.groups - 1) / A.groups;  // tiles in groups of one or two
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&s_tmem)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int i = 0; i < SLOTS; ++i) {
            mbar_init(full0 + 8 * i, 1);
            mbar_init(empty0 + 8 * i, 1);
        }
        for (int g = 0; g < 2; ++g) {
            mbar_init(ready0 + 8 * g, GROUP / 32);
            mbar_init(acc0 + 8 * g, 1);
        }
        mbar_init(drain, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    if (warp < 16) {
        // ---- a tile's features and epilogues
        const int g = warp >> 3, gt = tid & (GROUP - 1), gw = warp & 7;
        unsigned char* sA = smem + g * SMEM_A;
        const int row = gt & 127, half = gt >> 7;                                  // features: point row, 64-feature half
        const int erow = 32 * (gw & 3) + lane, ecol0 = 128 * (gw >> 2);            // epilogue
        const uint32_t taddr = tmem + (uint32_t)(256 * g) + ((uint32_t)(32 * (gw & 3)) << 16);
        uint32_t phase = 0;
        bool ok = g < (int)A.groups;
        for (uint64_t step = blockIdx.x; step < steps && ok; step += gridDim.x) {
            const uint64_t tile = step * A.groups + g, pidx = tile * 128 + row;
            float q[3] = {0.0f, 0.0f, 0.0f};
            if (pidx < A.n) point_of(A, pidx, q);
            write_features(sA, row, half, q);
            float y = 0.0f;
            for (int l = 0; l < NLAYERS; ++l) {
                // the operand is written and the accumulator read
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(ready0 + 8 * g);
                const float* bias = A.bias + l * HID;
                // one decision for the group: its barriers need every thread
                ok = group_all(g, mbar_wait(acc0 + 8 * g, phase, &s_abort));
                phase ^= 1;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // row erow, columns [ecol0, ecol0 + 128), 16 at a time; the
                // TMEM load of the next 16 overlaps the arithmetic on these
                uint32_t ra[16], rb[16];
                uint64_t sum = f2(0.0f, 0.0f);
                tmem_ld16(taddr + ecol0, ra);
                tmem_wait(ra);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint32_t(&cur)[16] = (c & 1) ? rb : ra;
                    uint32_t(&nxt)[16] = (c & 1) ? ra : rb;
                    const int c0 = ecol0 + 16 * c;
                    if (c + 1 < 8) tmem_ld16(taddr + c0 + 16, nxt);
                    uint64_t r[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        r[i] = softplus2(f2(__uint_as_float(cur[2 * i]), __uint_as_float(cur[2 * i + 1])),
                                         f2(bias[c0 + 2 * i], bias[c0 + 2 * i + 1]));
                    if (l + 1 < NLAYERS) {
                        uint32_t p[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float a0, a1;
                            uf2(r[i], a0, a1);
                            __nv_bfloat162 h = __floats2bfloat162_rn(a0, a1);
                            p[i] = *reinterpret_cast<uint32_t*>(&h);
                        }
                        *reinterpret_cast<uint4*>(sA + swz(erow, c0, 128)) = make_uint4(p[0], p[1], p[2], p[3]);
                        *reinterpret_cast<uint4*>(sA + swz(erow, c0 + 8, 128)) = make_uint4(p[4], p[5], p[6], p[7]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            sum = fma2(r[i], f2(A.wout[c0 + 2 * i], A.wout[c0 + 2 * i + 1]), sum);
                        }
                    }
                    if (c + 1 < 8) tmem_wait(nxt);
                }
                if (l + 1 == NLAYERS) {
                    float a0, a1;
                    uf2(sum, a0, a1);
                    y = a0 + a1;
                }
            }
            if (!ok) break;
            // output: the two column halves of each row
            if (ecol0) s_part[g][erow] = y;
            group_all(g, true);
            if (!ecol0) {
                const uint64_t o = tile * 128 + erow;
                if (o < A.n) A.out[o] = y + s_part[g][erow] + A.wout[HID];
            }
        }
        if (!ok && g < (int)A.groups) {
            s_abort = 1;
            if (gt == 0) atomicOr(A.err, DERR_QUEUE_TIMEOUT);
        }
    } else if (warp == 16 && lane == 0) {
        // ---- the tiles' layers in turn
        uint32_t phase = 0;   // both tiles' ready barriers move together
        uint32_t kbi = 0;     // K-blocks taken so far
        const uint64_t bdesc = sdesc(sB);
        bool ok = true;
        for (uint64_t step = blockIdx.x; step < steps && ok; step += gridDim.x) {
            for (int l = 0; l < NLAYERS && ok; ++l, phase ^= 1) {
                for (int g = 0; g < (int)A.groups && ok; ++g) {
                    ok = mbar_wait(ready0 + 8 * g, phase, &s_abort);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    // (descriptor addresses count 16 bytes: a K = 16 step is 2 on)
                    uint64_t ad = sdesc(smem_u32(smem + g * SMEM_A));
                    for (int kb = 0; kb < kblocks_of(l); ++kb, ++kbi) {
                        const uint32_t slot = kbi % SLOTS;
                        ok = mbar_wait(full0 + 8 * slot, (kbi / SLOTS) & 1u, &s_abort);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        const uint64_t bd = bdesc + slot * (uint32_t)(KBLOCK_BYTES_B >> 4);
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                            mma(tmem + (uint32_t)(256 * g), ad + 2 * s, bd + 2 * s, (kb | s) ? 1u : 0u);
                        ad += KBLOCK_BYTES_A >> 4;
                        commit_to(empty0 + 8 * slot);
                    }
                    if (ok) commit_to(acc0 + 8 * g);
                }
            }
        }
        if (!ok) {
            s_abort = 1;
            atomicOr(A.err, DERR_QUEUE_TIMEOUT);
        }
        // nothing issued here is still running when TMEM is freed
        commit_to(drain);
        mbar_wait(drain, 0, nullptr);
    } else if (warp == 17 && lane == 0) {
        // ---- weights: the K-blocks of the layers in the order the MMAs take them
        uint32_t kbi = 0;
        bool ok = true;
        for (uint64_t step = blockIdx.x; step < steps && ok; step += gridDim.x) {
            for (int l = 0; l < NLAYERS && ok; ++l) {
                const unsigned char* src = A.w + 2 * image_offset(l);
                for (int g = 0; g < (int)A.groups && ok; ++g) {
                    for (int kb = 0; kb < kblocks_of(l); ++kb, ++kbi) {
                        const uint32_t slot = kbi % SLOTS, bar = full0 + 8 * slot;
                        ok = mbar_wait(empty0 + 8 * slot, ((kbi / SLOTS) & 1u) ^ 1u, &s_abort);
                        if (!ok) break;
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar),
                                     "r"((uint32_t)KBLOCK_BYTES_B)
                                     : "memory");
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
                                "r"(sB + slot * (uint32_t)KBLOCK_BYTES_B),
                            "l"(src + kb * KBLOCK_BYTES_B), "r"((uint32_t)KBLOCK_BYTES_B), "r"(bar)
                            : "memory");
                    }
                }
            }
        }
        if (!ok) {
            s_abort = 1;
            atomicOr(A.err, DERR_QUEUE_TIMEOUT);
        }
        // the last copy into each slot has landed before the CTA ends
        for (uint32_t i = kbi > SLOTS ? kbi - SLOTS : 0; i < kbi; ++i)
            mbar_wait(full0 + 8 * (i % SLOTS), (i / SLOTS) & 1u, nullptr);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem));
}

}  // namespace

namespace iso {

static MlpImages* images_of(iso_mlp* net) {
    if (!net->infer) net->infer = new MlpImages();
    return (MlpImages*)net->infer;
}

void mlp_infer_release(iso_mlp* net) {
    MlpImages* m = (MlpImages*)net->infer;
    if (!m) return;
    if (m->w) cudaFree(m->w);
    delete m;
    net->infer = nullptr;
}

void mlp_infer_invalidate(iso_mlp* net, const float* params) {
    if (!net->infer && !params) return;
    MlpImages* m = images_of(net);
    m->valid = m->host_valid = false;
    if (!params) return;
    // what the kernel takes by value need not come back from the device
    m->host.resize(NLAYERS * HID + HID + 1);
    for (int l = 0; l < NLAYERS; ++l) std::copy_n(params + bias_offset(l), HID, m->host.begin() + l * HID);
    std::copy_n(params + OUT_W, HID + 1, m->host.begin() + NLAYERS * HID);
    m->host_valid = true;
}

static iso_status ready(iso_mlp* net, MlpImages** out) {
    iso_ctx* ctx = net->ctx;
    MlpImages* m = images_of(net);
    if (!m->w) {
        void* p = nullptr;
        cudaError_t e = cudaMalloc(&p, IMAGE_ELEMS * 2 + 4 * (NLAYERS * HID + HID + 1) + 256);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp images");
        m->w = (__nv_bfloat16*)p;
        m->bias = (float*)((char*)p + ((IMAGE_ELEMS * 2 + 255) & ~(size_t)255));
        m->wout = m->bias + NLAYERS * HID;
    }
    if (!m->valid) {
        prepare_images<<<(unsigned)((IMAGE_ELEMS + 255) / 256), 256, 0, ctx->stream>>>(net->params, m->w,
                                                                                     m->bias, m->wout);
        ctx->launches++;
        iso_status s = check_launch(ctx, "prepare images");
        if (s != ISO_OK) return s;
        if (!m->host_valid) {  // trained on the device
            m->host.resize(NLAYERS * HID + HID + 1);
            cudaError_t e = cudaMemcpyAsync(m->host.data(), m->bias, 4 * m->host.size(), cudaMemcpyDeviceToHost, ctx->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp biases");
            m->host_valid = true;
        }
        m->valid = true;
    }
    *out = m;
    return ISO_OK;
}

iso_status mlp_infer_launch(iso_mlp* net, const float* d_pts, uint64_t n, const MlpGrid* grid, float* d_out) {
    iso_ctx* ctx = net->ctx;
    MlpImages* m = nullptr;
    iso_status s = ready(net, &m);
    if (s != ISO_OK) return s;
    InferArgs a{};
    a.w = reinterpret_cast<const unsigned char*>(m->w);
    std::copy(m->host.begin(), m->host.begin() + NLAYERS * HID, a.bias);
    std::copy(m->host.begin() + NLAYERS * HID, m->host.end(), a.wout);
    a.pts = d_pts;
    a.n = n;
    if (grid) {
        a.nx = grid->nx;
        a.ny = grid->ny;
        a.nz = grid->nz;
        a.step = grid->step;
        a.inv = grid->inv;
        for (int i = 0; i < 3; ++i) {
            a.scale[i] = grid->scale[i];
            a.offset[i] = grid->offset[i];
        }
        a.n = (uint64_t)grid->nx * grid->ny * grid->nz;
    }
    a.out = d_out;
    a.err = ctx->d_err;
    cudaError_t e = cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_TOTAL);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp smem attribute");
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (a.n == 0) return ISO_OK;
    // two tiles per CTA once every SM has one
    const uint64_t tiles = (a.n + 127) / 128;
    a.groups = tiles > (uint64_t)sms ? 2 : 1;
    const unsigned blocks = (unsigned)std::min<uint64_t>((tiles + a.groups - 1) / a.groups, (uint64_t)sms);
    {
        StageTimer timer(ctx, ISO_STAGE_MLP);
        mlp_infer_kernel<<<blocks, THREADS, SMEM_TOTAL, ctx->stream>>>(a);
    }
    ctx->launches++;
    return check_launch(ctx, "mlp infer");
}

}  // namespace iso

extern "C" iso_status iso_mlp_forward_bf16(iso_mlp* net, const float* pts, uint32_t n, float* values) {
    if (!net || (!pts && n) || (!values && n)) return ISO_ERR_INVALID_ARG;
    if (n == 0) return ISO_OK;
    iso_ctx* ctx = net->ctx;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->aux, 16ull * n + 256)) != ISO_OK) return s;
    float* d_pts = (float*)ctx->aux.p;
    float* d_out = d_pts + 3ull * n;
    cudaError_t e = cudaMemcpyAsync(d_pts, pts, 12ull * n, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "upload points");
    if ((s = mlp_infer_launch(net, d_pts, n, nullptr, d_out)) != ISO_OK) return s;
    e = cudaMemcpyAsync(values, d_out, 4ull * n, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp bf16 forward");
    return read_device_errors(ctx);
}
