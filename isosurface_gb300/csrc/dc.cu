// DualContouring::new(size, placer).extract (src/dual_contouring.rs:65-105)
// over DualGrid::traverse (src/traversal/dual_grid.rs:52-95).
//
// The dual lattice has one vertex per primal cell: (size-1) x (size-1) x size
// vertices.  Its value is lerp(v0, v6, 0.5) of the primal corners
// (dual_grid.rs:80-81); its position is the cell centre lerp(c0, c6, 0.5)
// unless the cell is active (case not 0 or 255), where the feature placer
// puts it (dual_contouring.rs:78-87).  The dual cubes are then meshed exactly
// like MarchingCubes over the dual lattice with explicit vertex positions
// (dual_contouring.rs:88-101 is the same cell kernel with GridKey dedup), so
// the last two passes are mc_extract_lattice.
//
// Passes: (1) grid sampler (sign bits everywhere; for a program with a
// Lipschitz bound, values only near the surface), (2) dc_signs: dual sign
// words and the active primal cells, from the primal sign bits, (3) dc_edges:
// the active cells at an end of a crossing dual edge, and the values and
// centres that marching cubes reads there, (4) dc_place: one thread per
// such cell -- eight normals from the program (sample_normals_at_corners,
// marching_cubes_impl.rs:58-69), tangent planes, the planar cells' centre of
// mass or particle placement, the non-planar cells listed for (5) dc_feature:
// their MinimiseQEF (f64 SVD); (4) and (5) on a side stream
// beside (6) the lattice marching-cubes passes, whose emission waits for them.
// A program without a bound takes its full field through dc_dual in place of
// (2) and (3).
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"
#include "qef.cuh"
#include "qef_rows.cuh"
#include "vm.cuh"
#include "dc_core.cuh"

namespace iso {
// jit.cu: dc_place with the program's compiled normals; false (nothing
// launched) when the program has none
bool jit_dc_place(cudaStream_t stream, const iso_program* prog, const DcCells& cells, uint64_t blocks,
                  cudaError_t* err);

namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;

struct DualArgs {
    const float* field;   // primal values
    const uint32_t* bits; // primal sign bits (bit set iff !(v > 0)), W words per row
    uint32_t W;
    uint64_t pitch;       // primal row pitch
    uint32_t n;           // primal size: n x n x (n+1) samples
    uint32_t nzd;         // dual layers here (primal cell layers zoff .. zoff + nzd - 1)
    uint32_t zoff;        // primal cell layer of dual layer 0 (a slab of the whole lattice)
    float inv;
    float* dval;          // dual values, rows of dpitch
    uint64_t dpitch;
    float4* dpos;         // dual positions, dense (n-1) x (n-1) x nzd
    uint32_t* dbits;      // dual sign bits (bit set iff !(value > 0)), dW words per row
    uint32_t* abits;      // active primal cells, laid out as dbits
    uint32_t dW;
    uint32_t* list;       // active primal cells (linear dual index)
    uint32_t* count;
    uint32_t* ends;       // dc_edges: those at an end of a crossing dual edge
    uint32_t* nends;
    uint32_t cap;
    uint32_t* err;
    uint32_t run;         // dc_signs: layers per warp
};

// Vec3::lerp / Signed::lerp with f = 0.5: (1 - f) * a + f * b
__device__ __forceinline__ float half_lerp(float a, float b) {
    const float of = 1.0f - 0.5f;
    return of * a + 0.5f * b;
}

__device__ __forceinline__ float4 dual_centre(const DualArgs& A, uint32_t x, uint32_t y, uint32_t z) {
    const float c0x = (float)x * A.inv, c0y = (float)y * A.inv, c0z = (float)(z + A.zoff) * A.inv;
    const float c6x = (float)(x + 1) * A.inv, c6y = (float)(y + 1) * A.inv, c6z = (float)(z + 1 + A.zoff) * A.inv;
    return make_float4(half_lerp(c0x, c6x), half_lerp(c0y, c6y), half_lerp(c0z, c6z), 0.0f);
}

// corners 0 and 6 of dual vertex (x, y, z)'s primal cell
__device__ __forceinline__ void dual_corners(const DualArgs& A, uint32_t x, uint32_t y, uint32_t z, float* v0,
                                             float* v6) {
    const float* f0 = A.field + ((size_t)z * A.n + y) * A.pitch + x;
    *v0 = __ldg(f0);
    *v6 = __ldg(f0 + (size_t)A.n * A.pitch + A.pitch + 1);
}

// Dual sign words and active cells, from sign bits alone wherever the cell's
// corners 0 and 6 agree: the dual value, their mean, then has their sign
// (no program here produces values within an ulp of zero's neighbours, see
// iso_program::tiny).  Where they differ the surface passes between two points
// sqrt(3) lattice steps apart, so both lie within that of zero and the
// sampler (which keeps 2.5 steps) wrote them.  Lane = 32 dual vertices of a
// row; a warp marches its 32 words up `run` layers, the sign words of a layer
// serving the cells below and above it.  The active cells of a step are
// handed out one per lane.
__global__ void __launch_bounds__(256) dc_signs(DualArgs A) {
    __shared__ uint32_t s_word[8][32];
    const uint32_t m = A.n - 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t S = A.dW * m, SL = (S + 31) / 32;
    const uint32_t task = blockIdx.x * 8 + warp, seg = task % SL, z0 = task / SL * A.run;
    if (z0 >= A.nzd) return;  // warp-uniform
    const uint32_t l = 32 * seg + lane, y = l / A.dW, c = l - y * A.dW;
    const bool in = l < S, nxt = in && c + 1 < A.W;
    const uint32_t left = in ? m - 32 * c : 0u;
    const uint32_t valid = left >= 32 ? FULL : (1u << left) - 1u;
    const uint64_t layer = (uint64_t)A.n * A.W;
    const uint32_t* p = A.bits + z0 * layer + (uint64_t)y * A.W + c;
    auto quad = [&](const uint32_t* q) {  // corners (x,y) (x+1,y) (x+1,y+1) (x,y+1)
        const uint32_t a0 = in ? __ldg(q) : 0u, an = nxt ? __ldg(q + 1) : 0u;
        const uint32_t b0 = in ? __ldg(q + A.W) : 0u, bn = nxt ? __ldg(q + A.W + 1) : 0u;
        return make_uint4(a0, __funnelshift_r(a0, an, 1), __funnelshift_r(b0, bn, 1), b0);
    };
    uint4 lo = quad(p);
    const uint32_t z1 = min(z0 + A.run, A.nzd);
    for (uint32_t z = z0; z < z1; ++z) {
        p += layer;
        const uint4 hi = quad(p);
        const uint32_t any = lo.x | lo.y | lo.z | lo.w | hi.x | hi.y | hi.z | hi.w;
        const uint32_t all = lo.x & lo.y & lo.z & lo.w & hi.x & hi.y & hi.z & hi.w;
        const uint32_t act = any & ~all & valid, diff = (lo.x ^ hi.z) & valid;
        uint32_t word = lo.x & hi.z & valid;
        if (__any_sync(FULL, act != 0)) {
            const uint32_t n = __popc(act);
            uint32_t incl = n;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            const uint32_t excl = incl - n, total = __shfl_sync(FULL, incl, 31);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(A.count, total);
            base = __shfl_sync(FULL, base, 0);
            s_word[warp][lane] = word;
            __syncwarp();
            for (uint32_t b0 = 0; b0 < total; b0 += 32) {
                const uint32_t kk = b0 + lane;
                uint32_t src = 0;  // the last lane whose prefix is <= kk
#pragma unroll
                for (uint32_t step = 16; step > 0; step >>= 1) {
                    const uint32_t e = __shfl_sync(FULL, excl, (src + step) & 31);
                    if (src + step < 32 && e <= kk) src += step;
                }
                uint32_t bits = __shfl_sync(FULL, act, src), r = kk - __shfl_sync(FULL, excl, src), i = 0;
                const uint32_t dsrc = __shfl_sync(FULL, diff, src), lsrc = __shfl_sync(FULL, lo.x, src);
                const uint32_t ysrc = __shfl_sync(FULL, y, src), csrc = __shfl_sync(FULL, c, src);
                if (kk >= total) continue;
#pragma unroll
                for (uint32_t w = 16; w > 0; w >>= 1) {  // set bit number r
                    const uint32_t below = __popc(bits & ((1u << w) - 1u));
                    if (r >= below) {
                        r -= below;
                        bits >>= w;
                        i += w;
                    }
                }
                const uint32_t x = 32 * csrc + i;
                if (base + kk < A.cap) A.list[base + kk] = (uint32_t)(((uint64_t)z * m + ysrc) * m + x);
                else atomicOr(A.err, DERR_CAPACITY);
                if ((dsrc >> i) & 1u) {
                    float v0, v6;
                    dual_corners(A, x, ysrc, z, &v0, &v6);
                    const bool inside = v0 == v0 && v6 == v6 ? !(half_lerp(v0, v6) > 0.0f) : (lsrc >> i) & 1u;
                    if (inside) atomicOr(&s_word[warp][src], 1u << i);
                }
            }
            __syncwarp();
            word = s_word[warp][lane];
            __syncwarp();
        }
        if (in) {
            const uint64_t at = ((uint64_t)z * m + y) * A.dW + c;
            A.dbits[at] = word;
            A.abits[at] = act;
        }
        lo = hi;
    }
}

// One thread per active cell: marching cubes reads the value and position of
// a dual vertex only at the ends of crossing dual edges, and of the two ends
// at least one belongs to an active cell (cells that share four corners and
// have no sign change have the same sign).  An active cell with such an edge
// gets its value here and its position from the placement; its inactive
// neighbours across such edges get their value and cell centre here.
__global__ void __launch_bounds__(256) dc_edges(DualArgs A) {
    const uint32_t m = A.n - 1, lane = threadIdx.x & 31, n = *A.count;
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        bool end = false;
        uint32_t id = 0;
        if (i < n) {
            id = A.list[i];
            const uint32_t x = id % m, r = id / m, y = r % m, z = r / m;
            auto bit = [&](const uint32_t* words, uint32_t xx, uint32_t yy, uint32_t zz) {
                return (__ldg(words + ((uint64_t)zz * m + yy) * A.dW + (xx >> 5)) >> (xx & 31)) & 1u;
            };
            const uint32_t own = bit(A.dbits, x, y, z);
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const uint32_t axis = k >> 1, up = k & 1;
                const uint32_t at = axis == 0 ? x : axis == 1 ? y : z, lim = axis == 2 ? A.nzd : m;
                if (up ? at + 1 >= lim : at == 0) continue;
                const uint32_t d = up ? 1u : 0xFFFFFFFFu;
                const uint32_t xx = x + (axis == 0 ? d : 0u), yy = y + (axis == 1 ? d : 0u), zz = z + (axis == 2 ? d : 0u);
                if (bit(A.dbits, xx, yy, zz) == own) continue;
                end = true;
                if (bit(A.abits, xx, yy, zz)) continue;  // it looks after itself
                float v0, v6;
                dual_corners(A, xx, yy, zz, &v0, &v6);
                A.dval[((size_t)zz * m + yy) * A.dpitch + xx] = half_lerp(v0, v6);
                A.dpos[((uint64_t)zz * m + yy) * m + xx] = dual_centre(A, xx, yy, zz);
            }
            if (end) {
                float v0, v6;
                dual_corners(A, x, y, z, &v0, &v6);
                A.dval[((size_t)z * m + y) * A.dpitch + x] = half_lerp(v0, v6);
            }
        }
        const uint32_t mask = __ballot_sync(FULL, end);
        if (mask) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(A.nends, (uint32_t)__popc(mask));
            base = __shfl_sync(FULL, base, 0);
            if (end) A.ends[base + __popc(mask & ((1u << lane) - 1u))] = id;
        }
    }
}

// A full field (every value sampled): one warp per 32 dual vertices of a dual
// row (x = 32 w + lane): value, centre, sign word (by ballot) and the active
// primal cells.
__global__ void __launch_bounds__(256) dc_dual(DualArgs A) {
    const uint32_t m = A.n - 1, lane = threadIdx.x & 31;
    const uint64_t gw = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (gw >= (uint64_t)A.dW * m * A.nzd) return;  // warp-uniform
    const uint32_t w = (uint32_t)(gw % A.dW);
    const uint64_t row = gw / A.dW;
    const uint32_t y = (uint32_t)(row % m), z = (uint32_t)(row / m);
    const uint32_t x = 32 * w + lane;
    bool active = false, inside = false;
    if (x < m) {
        // corner signs from the sign bits, in CORNERS order (marching_cubes_tables.rs:16-25)
        auto sign_bit = [&](uint32_t xx, uint32_t yy, uint32_t zz) {
            return (__ldg(A.bits + ((size_t)zz * A.n + yy) * A.W + (xx >> 5)) >> (xx & 31)) & 1u;
        };
        const uint32_t cs = sign_bit(x, y, z) | sign_bit(x + 1, y, z) << 1 | sign_bit(x + 1, y + 1, z) << 2 |
                            sign_bit(x, y + 1, z) << 3 | sign_bit(x, y, z + 1) << 4 |
                            sign_bit(x + 1, y, z + 1) << 5 | sign_bit(x + 1, y + 1, z + 1) << 6 |
                            sign_bit(x, y + 1, z + 1) << 7;
        float v0, v6;
        dual_corners(A, x, y, z, &v0, &v6);
        // the field's own NaN gets a signed sentinel in its place
        const float dv = v0 == v0 && v6 == v6 ? half_lerp(v0, v6) : ((cs & 1u) ? -3.0e38f : 3.0e38f);
        A.dpos[((uint64_t)z * m + y) * m + x] = dual_centre(A, x, y, z);
        A.dval[((size_t)z * m + y) * A.dpitch + x] = dv;
        inside = !(dv > 0.0f);
        active = cs != 0 && cs != 255;
    }
    const uint32_t word = __ballot_sync(FULL, inside);
    if (lane == 0) A.dbits[row * A.dW + w] = word;
    // warp-aggregated append of the active cells (their order does not matter)
    const uint32_t mask = __ballot_sync(FULL, active);
    if (mask) {
        uint32_t base = 0;
        if (lane == (uint32_t)__ffs(mask) - 1) base = atomicAdd(A.count, (uint32_t)__popc(mask));
        base = __shfl_sync(FULL, base, __ffs(mask) - 1);
        if (active) {
            const uint32_t at = base + __popc(mask & ((1u << lane) - 1u));
            if (at < A.cap) A.list[at] = (uint32_t)(((uint64_t)z * m + y) * m + x);
            else atomicOr(A.err, DERR_CAPACITY);
        }
    }
}

// The interpreter's normals (eval_hermite) as a dc_core.cuh evaluator.
struct VmHermite {
    ProgView pv;
    __device__ __forceinline__ V3 normal(V3 p) const {
        V3 nn;
        eval_hermite(pv, p, &nn);
        return nn;
    }
};

__global__ void __launch_bounds__(128) dc_place(VmHermite ev, DcCells A) { dc_place_body(ev, A); }

// MinimiseQEF of feature cell i (its normals kept) by the eight lanes of
// `mask`, a corner each: tangent_planes, then the solve.
__device__ __forceinline__ void feature_by_rows(const DcCells& A, uint32_t i, uint32_t mask, uint32_t* err) {
    using namespace qef;
    const uint32_t y = threadIdx.x & 7, id = A.features[i], m = A.n - 1;
    const uint32_t cx = id % m, r = id / m, cy = r % m, cz = r / m + A.zoff;
    const float px[2] = {(float)cx * A.inv, (float)(cx + 1) * A.inv};
    const float py[2] = {(float)cy * A.inv, (float)(cy + 1) * A.inv};
    const float pz[2] = {(float)cz * A.inv, (float)(cz + 1) * A.inv};
    // corner k of CORNERS (marching_cubes_tables.rs:16-25)
    auto corner = [&](uint32_t k) { return f3(px[(k + 1) >> 1 & 1], py[k >> 1 & 1], pz[k >> 2]); };
    const F3 nrm = A.fnormals[8 * (uint64_t)i + y];
    auto normal_of = [&](uint32_t k) {
        return f3(__shfl_sync(mask, nrm.x, k, 8), __shfl_sync(mask, nrm.y, k, 8), __shfl_sync(mask, nrm.z, k, 8));
    };
    F3 com = f3(0.0f, 0.0f, 0.0f);
    float least = 3.40282347e+38f;
    uint32_t pair = ~0u;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        com = add(com, corner(k));
        const float angle = dot(nrm, normal_of(k));
        if (angle < least) {
            least = angle;
            pair = 8 * y + k;
        }
    }
    com = f3(com.x / 8.0f, com.y / 8.0f, com.z / 8.0f);
    for (uint32_t o = 1; o < 8; o <<= 1) {  // the first of equals in (i, j) order
        const float a = __shfl_xor_sync(mask, least, o, 8);
        const uint32_t q = __shfl_xor_sync(mask, pair, o, 8);
        if (a < least || (a == least && q < pair)) {
            least = a;
            pair = q;
        }
    }
    F3 p = com;
    bool ok = true;
    if (!(least > FEATURE_ANGLE)) {
        const F3 na = normal_of(pair >> 3 & 7), nb = normal_of(pair & 7);
        const F3 axis = normalised_or_zero(pair == ~0u ? f3(0.0f, 0.0f, 0.0f) : cross(na, nb));
        const float along = dot(axis, nrm);
        float lo = fminf(1.0f, along), hi = fmaxf(-1.0f, along);
        for (uint32_t o = 1; o < 8; o <<= 1) {
            lo = fminf(lo, __shfl_xor_sync(mask, lo, o, 8));
            hi = fmaxf(hi, __shfl_xor_sync(mask, hi, o, 8));
        }
        float c = fmaxf(fabsf(lo), fabsf(hi));
        c = sqrtf(1.0f - c * c);
        p = add(com, solve_planes_rows(mask, nrm, dot(sub(corner(y), com), nrm), 8, c > FEATURE_ANGLE, &ok));
    }
    if (y != 0) return;
    if (!ok) atomicOr(err, DERR_SVD_ITER);
    A.dpos[id] = DcPos{p.x, p.y, p.z, 0.0f};
}

// MinimiseQEF of the non-planar cells dc_place listed, over one-warp blocks,
// six to an SM.  A solve is a serial
// chain of f64 operations (the SVD, in the reference's order), and a warp's
// f64 instruction holds its sub-partition's unit for many cycles however few
// of its lanes are active.  Few cells go to eight lanes each (qef_rows.cuh),
// which shortens the chain; more, beyond six warps of four cells per SM, to
// one lane each, in full warps, which issues fewer instructions (csg at 65:
// 163 us with six, 180 with four; more is no faster).  257 lattice, about 10000 cells: 121 us with a lane each (138
// with its matrices in local memory), 175 with four lanes each.  Two kernels,
// of which one has nothing to do: in one, the one-lane solve took 131 us.
constexpr uint32_t ROW_WARPS = 6;  // one-warp blocks per SM
__device__ __forceinline__ bool by_rows(const DcCells& A, uint32_t n, uint32_t blocks) {
    return n <= A.fcap && n <= 4 * blocks;
}

__global__ void __launch_bounds__(32) dc_feature_rows(DcCells A, uint32_t* err) {
    const uint32_t n = *A.nfeatures, group = threadIdx.x >> 3, i = 4 * blockIdx.x + group;
    if (by_rows(A, n, gridDim.x) && i < n) feature_by_rows(A, i, 0xFFu << (8 * group), err);
}

__global__ void __launch_bounds__(32) dc_feature(VmHermite ev, DcCells A, uint32_t* err) {
    const uint32_t n = *A.nfeatures;
    if (by_rows(A, n, gridDim.x)) return;
    for (uint32_t i = blockIdx.x * 32 + threadIdx.x; i < n; i += gridDim.x * 32) {
        const uint32_t id = A.features[i];
        qef::F3 corners[8], normals[8];
        if (i < A.fcap) {  // the normals dc_place computed when it listed the cell
            const uint32_t m = A.n - 1;
            const uint32_t x = id % m, r = id / m, y = r % m, z = r / m;
            const uint8_t cornr[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                         {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
            for (int k = 0; k < 8; ++k) {
                corners[k] = qef::f3((float)(x + cornr[k][0]) * A.inv, (float)(y + cornr[k][1]) * A.inv,
                                     (float)(z + A.zoff + cornr[k][2]) * A.inv);
                normals[k] = A.fnormals[8 * (uint64_t)i + k];
            }
        } else {
            dc_cell_normals(ev, A, id, corners, normals);
        }
        qef::Planes t;
        qef::tangent_planes(corners, normals, &t);
        bool ok;
        const qef::F3 p = qef::minimise_qef(t, &ok);
        if (!ok) atomicOr(err, DERR_SVD_ITER);
        A.dpos[id] = DcPos{p.x, p.y, p.z, 0.0f};
    }
}

}  // namespace
}  // namespace iso

using namespace iso;

static iso_status dc_check(iso_ctx* ctx, const iso_program* prog, uint32_t size, uint32_t placer, uint32_t flags) {
    if (!ctx || !prog) return ISO_ERR_INVALID_ARG;
    if (prog->ctx != ctx) return fail(ctx, ISO_ERR_INVALID_ARG, "program belongs to another context");
    if (size == 0 || size > 16384) return fail(ctx, ISO_ERR_INVALID_ARG, "size out of range");
    if (placer > 1) return fail(ctx, ISO_ERR_INVALID_ARG, "placer must be 0 (MinimiseQEF) or 1 (particles)");
    if (flags & ~(uint32_t)ISO_FLAG_KEYS) return fail(ctx, ISO_ERR_INVALID_ARG, "unsupported flags");
    if ((uint64_t)(size - 1) * (size - 1) * size >= 0xFFFFFFFFull) return fail(ctx, ISO_ERR_TOO_LARGE, "grid too large");
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    ctx->last = iso_mesh_info{};
    ctx->last_flags = flags;
    ctx->last_vertex_floats = 3;
    return ISO_OK;
}

// The dual lattice's layers [zlo, zlo + nzd) of DualContouring::new(n) (dual
// layer k: one vertex per primal cell of cell layer k), from the primal
// sample layers [zlo, zlo + nzd]: values, signs and placed positions in the
// whole lattice's frame.  The whole extraction is zlo = 0, nzd = n.
static iso_status dc_lattice(iso_ctx* ctx, const iso_program* prog, uint32_t n, uint32_t placer, uint32_t zlo,
                             uint32_t nzd, Lattice* L) {
    const uint32_t m = n - 1, nzp = nzd + 1;  // primal sample layers
    const uint64_t pitch = default_pitch(n), W = words_per_row(n);
    const uint64_t ndual = (uint64_t)m * m * nzd;
    const uint64_t dpitch = default_pitch(m), dW = words_per_row(m);
    iso_status s;
    // primal field + bits | dual values | dual positions | dual bits, active
    // bits, counts, active list, end list, features' normals
    if ((s = ensure(ctx, ctx->field, 4ull * pitch * n * nzp)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->bits, 4ull * W * n * nzp)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->aux, 4ull * dpitch * m * nzd)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->aux2, 16ull * ndual)) != ISO_OK) return s;
    const uint64_t list_words = (ndual + 63) & ~(uint64_t)63, dwords = (dW * m * nzd + 63) & ~(uint64_t)63;
    // normals kept for the first feature cells (96 bytes each, at most 96 MB)
    const uint32_t fcap = (uint32_t)std::min<uint64_t>(list_words, 1u << 20);
    if ((s = ensure(ctx, ctx->aux3, 8ull * dwords + 8ull * list_words + 256 + 96ull * fcap)) != ISO_OK) return s;
    float* field = (float*)ctx->field.p;
    uint32_t* bits = (uint32_t*)ctx->bits.p;
    float* dval = (float*)ctx->aux.p;
    float4* dpos = (float4*)ctx->aux2.p;
    uint32_t* dbits = (uint32_t*)ctx->aux3.p;
    uint32_t* abits = dbits + dwords;
    uint32_t* count = abits + dwords;  // active cells, then those at crossing edges, then the non-planar ones
    uint32_t* list = count + 64;
    uint32_t* ends = list + list_words;
    qef::F3* fnormals = reinterpret_cast<qef::F3*>(ends + list_words);
    const float inv = 1.0f / (float)(n - 1);
    // values only near the surface (programs with a Lipschitz bound): the
    // dual values read the primal ones up to 1 + sqrt(3)/2 lattice steps'
    // worth of change from zero (a dual crossing end within one step's
    // worth, and half the cell diagonal between its two corners); the
    // sampler keeps 2.5
    const bool near = prog->lip > 0.0f && !prog->tiny;
    if ((s = launch_sample_grid(ctx, prog, n, n, nzp, inv, field, pitch, bits, near, zlo, 2.5f)) != ISO_OK) return s;
    cudaError_t e = cudaMemsetAsync(count, 0, 12, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "memset");
    const uint64_t sms = (uint64_t)std::max(ctx->sms, 1);
    DualArgs da{field, bits, (uint32_t)W, pitch, n, nzd, zlo, inv, dval, dpitch, dpos, dbits, abits, (uint32_t)dW,
                list, count, ends, count + 1, (uint32_t)ndual, ctx->d_err, 1};
    // the cells to place; the features' list takes the place of the one the placement does not read
    DcCells cells{n, zlo, inv, ends, count + 1, reinterpret_cast<DcPos*>(dpos), (int)placer, list, count + 2, fnormals,
                  fcap};
    StageTimer timer(ctx, ISO_STAGE_PLACE);
    if (near) {
        const uint64_t SL = (dW * m + 31) / 32;
        // as mc_cell_count: long runs share sign words, short ones keep the warps many
        da.run = (uint32_t)std::min<uint64_t>(16, std::max<uint64_t>(1, SL * nzd / (160 * sms)));
        const uint64_t warps = SL * ((nzd + da.run - 1) / da.run);
        dc_signs<<<(unsigned)((warps + 7) / 8), 256, 0, ctx->stream>>>(da);
        dc_edges<<<(unsigned)std::min<uint64_t>((ndual + 255) / 256, 8 * sms), 256, 0, ctx->stream>>>(da);
        ctx->launches++;
    } else {
        const uint64_t dual_warps = dW * m * nzd;
        dc_dual<<<(unsigned)((dual_warps + 7) / 8), 256, 0, ctx->stream>>>(da);
        cells.list = list;
        cells.count = count;
        cells.features = ends;
    }
    // placement on the side stream: only the mesh's vertices wait for it
    // (count and scan of a 256^3 lattice, 17 us, run beside it)
    cudaStream_t side;
    if ((s = fork_side(ctx, &side)) != ISO_OK) return s;
    timer.ends_on(side);
    const VmHermite ev{prog->view()};
    const uint64_t place_blocks = std::min<uint64_t>((ndual + 127) / 128, 152 * 64);
    cudaError_t je = cudaSuccess;
    if (!jit_dc_place(side, prog, cells, place_blocks, &je))  // the program's compiled normals (jit.cu)
        dc_place<<<(unsigned)place_blocks, 128, 0, side>>>(ev, cells);
    if (placer == 0 && je == cudaSuccess) {
        dc_feature_rows<<<(unsigned)(ROW_WARPS * sms), 32, 0, side>>>(cells, ctx->d_err);
        dc_feature<<<(unsigned)(ROW_WARPS * sms), 32, 0, side>>>(ev, cells, ctx->d_err);
        ctx->launches += 2;
    }
    ctx->launches += 2;
    if (je != cudaSuccess || (s = check_launch(ctx, "dc passes")) != ISO_OK) {
        join_side(ctx);
        return je != cudaSuccess ? cuda_fail(ctx, je, "compiled dc_place launch") : s;
    }
    *L = Lattice{m, m, nzd, dpitch, dval, dbits, (uint32_t)dW, 0.0f, dpos, zlo};
    L->join = true;
    return ISO_OK;
}

// marching cubes over the dual lattice; the side stream's placement is always
// joined, also when the passes end early
static iso_status dc_mesh(iso_ctx* ctx, const Lattice& L, uint32_t flags, iso_mesh_info* info) {
    const iso_status s = mc_extract_lattice(ctx, L, flags, info);
    if (ctx->side_open) {
        const iso_status j = join_side(ctx);
        if (s == ISO_OK) return j;
    }
    return s;
}

static iso_status dc_extract_impl(iso_ctx* ctx, const iso_program* prog, uint32_t size, uint32_t placer,
                                     uint32_t flags, iso_mesh_info* info) {
    iso_status s = dc_check(ctx, prog, size, placer, flags);
    if (s != ISO_OK) return s;
    if (size < 3) {  // the dual lattice has no cube
        if (info) *info = ctx->last;
        return ISO_OK;
    }
    Lattice L;
    if ((s = dc_lattice(ctx, prog, size, placer, 0, size, &L)) != ISO_OK) return s;
    return dc_mesh(ctx, L, flags, info);
}

// One slab of a z-partition of DualContouring::new(size): dual cube layers
// [z_begin, z_end) of the size - 1, plus the halo cube layer below when
// z_begin > 0, exactly as mc_extract_slab does for MarchingCubes.
extern "C" iso_status iso_dc_extract_slab(iso_ctx* ctx, const iso_program* prog, uint32_t size, uint32_t placer,
                                          uint32_t z_begin, uint32_t z_end, uint32_t flags, iso_mesh_info* info,
                                          uint64_t* halo_vertices, uint64_t* halo_triangles) {
    iso::NvtxRange nvtx_range("iso_dc_extract_slab");
    iso_status s = dc_check(ctx, prog, size, placer, flags);
    if (s != ISO_OK) return s;
    if (size < 3 || z_begin >= z_end || z_end > size - 1)
        return fail(ctx, ISO_ERR_INVALID_ARG, "need size >= 3 and 0 <= z_begin < z_end <= size - 1");
    const uint32_t halo = z_begin > 0 ? 1u : 0u, zlo = z_begin - halo;
    Lattice L;
    if ((s = dc_lattice(ctx, prog, size, placer, zlo, z_end - zlo + 1, &L)) != ISO_OK) return s;
    uint64_t hv = 0, ht = 0;
    if (halo && (s = mc_first_layer_counts(ctx, L, &hv, &ht)) != ISO_OK) {
        join_side(ctx);
        return s;
    }
    if ((s = dc_mesh(ctx, L, flags, info)) != ISO_OK) return s;
    if (halo_vertices) *halo_vertices = hv;
    if (halo_triangles) *halo_triangles = ht;
    return ISO_OK;
}

// ISO_FLAG_NORMALS: the *InterleavedNormals sinks, sample_normal at every vertex
extern "C" iso_status iso_dc_extract(iso_ctx* ctx, const iso_program* prog, uint32_t size, uint32_t placer, uint32_t flags, iso_mesh_info* info) {
    iso::NvtxRange nvtx_range("iso_dc_extract");
    if (!ctx || !prog) return ISO_ERR_INVALID_ARG;
    if (flags & ~(uint32_t)(ISO_FLAG_KEYS | ISO_FLAG_NORMALS)) return fail(ctx, ISO_ERR_INVALID_ARG, "unsupported flags");
    iso_status s = dc_extract_impl(ctx, prog, size, placer, flags & ~(uint32_t)ISO_FLAG_NORMALS, info);
    if (s != ISO_OK || !(flags & ISO_FLAG_NORMALS)) return s;
    return attach_normals(ctx, prog);
}
