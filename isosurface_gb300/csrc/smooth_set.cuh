// Culled sampling of a smooth union of many spheres (a SPHERE_SET with k > 0,
// optionally behind a domain map) for the extractors; included by sample.cu.
//
// The fold v = smooth_min(v, d_i, k) over the spheres in order returns one
// operand's bits unchanged wherever the operands differ by k or more.  So
// over a box of sample points on which every d_i lies in [lb_i, ub_i]:
//   * skip:  v <= min_{j<i} ub_j, so a sphere with lb_i >= that minimum + k
//            leaves v as it is at every point of the box;
//   * reset: a fold over values >= X stays above X - k (each step lowers v
//            by (k - |v - d|)^2 / 4k, which shrinks to nothing as v nears
//            X - k), so a sphere with ub_i + 2k <= min_{j<i} lb_j replaces v
//            by d_i at every point of the box: the fold may start there.
// Where the partial fold's own value at the box's centre is known, its value
// over the box (it is as Lipschitz as the spheres) takes those bounds' place.
// The fold from the last reset over the spheres not skipped therefore gives
// the full fold's bits.  k is widened by the rounding slack in both tests.
//
// A brute sample costs n sphere evaluations; here three levels share them:
//   smooth_boxes     one block per box (32 samples along x, `rows` along y and
//                    z): the box's sphere list from all n;
//   smooth_classify  one thread per 8 x 4 x 4 sub-brick: its spheres out of the
//                    box's list as a bit mask, and its class from the value
//                    at its centre (bricks_core.cuh's rule: wholly beyond
//                    reach of the surface -> sign bits only);
//   smooth_rows      one warp per mixed sub-brick, four samples per lane: the
//                    exact fold over its spheres.
// All three are bound by issue slots (roots, comparisons and the smooth
// minimum's division).  4096 spheres of radius 0.01-0.08, k = 0.05, at 257^3:
// 0.055 + 0.054 + 0.34 ms, against 1.4 + 72 ms for the general culled sampler,
// which folds every sphere at each sub-brick's centre and at each sample of
// the mixed ones.  Boxes by a whole block rather than a warp: 0.07 against
// 0.09 ms; the root left out where the squared distance decides, and compact
// lanes in smooth_rows: 0.38 against 0.6 ms; the quotient by the width from
// its reciprocal: 0.34 against 0.39 ms.
#pragma once

namespace iso {
namespace {

constexpr uint32_t SMOOTH_ALL = 0xFFFFFFFFu;  // a list that outgrew its room: every sphere
constexpr uint32_t SMOOTH_MAX = 65535;        // spheres a 16-bit index reaches

struct SmoothArgs {
    const float4* sp;  // (centre, radius)
    uint32_t n;
    float k, kpad;  // smooth-min width; widened by the rounding of the bounds and of the fold
    float rk;       // 1 / k rounded to nearest, 0 where smooth_min_by does not apply
    bool domain;
    float sx, sy, sz, ox, oy, oz;
    BrickLattice g;
    uint32_t rows;    // samples per box along y and z: 16, 8 or 4
    uint32_t by, bz;  // boxes along y and z (g.W along x)
    uint32_t cap;     // list entries per box, a multiple of 32
    uint32_t nsub;    // sub-bricks per box
    uint32_t* len;    // per box: list length, 0 (decided) or SMOOTH_ALL
    uint16_t* list;   // per box: cap sphere indices, ascending
    uint32_t* mask;   // per box: cap / 32 words x nsub sub-bricks, bit = kept list position
    uint2* tasks;     // mixed sub-bricks: (box * nsub + sub-brick, list position the fold starts at)
    uint32_t* ntasks;
};

__device__ __forceinline__ V3 smooth_point(const SmoothArgs& A, V3 p) {
    return A.domain ? v3(p.x * A.sx + A.ox, p.y * A.sy + A.oy, p.z * A.sz + A.oz) : p;
}

// smooth_min for the one width k of a set.  The quotient gap / k is IEEE's:
// by Markstein's theorem (Computation of elementary functions on the IBM RISC
// System/6000 processor, 1990) a quotient within an ulp, corrected once by
// its exact remainder times the correctly rounded reciprocal, is correctly
// rounded.  The first correction gets it within the ulp, the second is the
// theorem's.  A gap is at least a rounding unit of k, so for widths from 2^-60
// to 2^60 (RK) nothing underflows.
template <bool RK>
__device__ __forceinline__ float smooth_min_by(float a, float b, float k, float rk) {
    if (!RK) return smooth_min(a, b, k);
    const float gap = k - fabsf(a - b), m = fminf(a, b);
    float h = gap * rk;
    h = __fmaf_rn(__fmaf_rn(-k, h, gap), rk, h);
    h = __fmaf_rn(__fmaf_rn(-k, h, gap), rk, h);
    // without overlap the formula gives min(a, b) - 0, as smooth_min does
    return gap > 0.0f ? m - ((h * h) * k) * 0.25f : m;
}

// centre of the samples [x0, x1] x [y0, y1] x [z0, z1] and a bound on the
// change of any sphere's value (or the union's) from there, rounding included
__device__ __forceinline__ float smooth_spread(const SmoothArgs& A, uint32_t x0, uint32_t x1, uint32_t y0, uint32_t y1,
                                               uint32_t z0, uint32_t z1, V3* c) {
    const BrickLattice& g = A.g;
    const float hx = 0.5f * (float)(x1 - x0), hy = 0.5f * (float)(y1 - y0), hz = 0.5f * (float)(z1 - z0);
    *c = smooth_point(A, v3(((float)x0 + hx) * g.inv, ((float)y0 + hy) * g.inv, ((float)(z0 + g.zoff) + hz) * g.inv));
    return g.lip * sqrtf((hx * hx + hy * hy) + hz * hz) * g.inv * (1.0f + 1.0f / 1024.0f) + g.slack;
}

__device__ __forceinline__ float smooth_reach(const BrickLattice& g) {
    return g.lip * g.inv * g.reach_steps * (1.0f + 1.0f / 1024.0f) + g.slack;
}

struct SmoothBox {
    uint32_t wx, y0, y1, z0, z1;  // rows [y0, y1), layers [z0, z1)
};

__device__ __forceinline__ SmoothBox smooth_box(const SmoothArgs& A, uint32_t box) {
    SmoothBox b;
    b.wx = box % A.g.W;
    const uint32_t r = box / A.g.W;
    b.y0 = (r % A.by) * A.rows;
    b.z0 = (r / A.by) * A.rows;
    b.y1 = min(b.y0 + A.rows, A.g.ny);
    b.z1 = min(b.z0 + A.rows, A.g.nz);
    return b;
}

__device__ __forceinline__ float warp_incl_min(float v, uint32_t lane) {
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v = fminf(v, t);
    }
    return v;
}

// One block per box.  The tests at sphere i need minima over the spheres
// before it, so its eight warps take consecutive ranges of the spheres and
// go over them three times with block-wide minima in between: the range's
// lowest lb; the last reset in it; the kept spheres after the last reset of
// all (as ballots in shared memory, then written out in order).
__global__ void __launch_bounds__(256) smooth_boxes(SmoothArgs A) {
    const float INF = __int_as_float(0x7F800000);
    __shared__ float s_low[8], s_up[8], s_since[8];
    __shared__ uint32_t s_reset[8], s_cnt[8];
    __shared__ uint32_t s_keep[8][SMOOTH_MAX / 256 + 1];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, box = blockIdx.x;
    const SmoothBox b = smooth_box(A, box);
    V3 c;
    const float spread = smooth_spread(A, 32 * b.wx, min(32 * b.wx + 31, A.g.nx - 1), b.y0, b.y1 - 1, b.z0, b.z1 - 1, &c);
    const uint32_t steps = (A.n + 255) / 256, i0 = warp * steps * 32 + lane;  // this warp: steps x 32 spheres
    auto value = [&](uint32_t i) {
        if (i >= A.n) return INF;
        const float4 s = __ldg(A.sp + i);
        return vlen(v3(c.x - s.x, c.y - s.y, c.z - s.z)) - s.w;
    };
    // the values of the first spheres stay in registers for all three rounds
    // (4096 spheres at 257^3: 68 us with each round computing its own)
    constexpr uint32_t HELD = 16;
    float held[HELD];
#pragma unroll
    for (uint32_t t = 0; t < HELD; ++t) held[t] = t < steps ? value(i0 + 32 * t) : INF;
    auto each = [&](auto&& f) {
#pragma unroll
        for (uint32_t t = 0; t < HELD; ++t)
            if (t < steps) f(t, held[t]);
        for (uint32_t t = HELD; t < steps; ++t) f(t, value(i0 + 32 * t));
    };
    float near = INF;
    each([&](uint32_t, float d) { near = fminf(near, d); });
    for (int o = 16; o > 0; o >>= 1) near = fminf(near, __shfl_xor_sync(0xFFFFFFFFu, near, o));
    if (lane == 0) {
        s_low[warp] = near - spread;
        s_up[warp] = near + spread;
    }
    __syncthreads();
    float low = INF, all_low = INF, all_up = INF;
    for (uint32_t w = 0; w < 8; ++w) {
        if (w < warp) low = fminf(low, s_low[w]);
        all_low = fminf(all_low, s_low[w]);
        all_up = fminf(all_up, s_up[w]);
    }
    // the union lies in [all_low - k, all_up] over the box
    const float reach = smooth_reach(A.g);
    const bool out = all_low - A.kpad > reach, in = all_up < -reach;
    if (out || in) {  // block-uniform
        const uint32_t valid = A.g.nx - 32 * b.wx;
        const uint32_t word = in ? (valid < 32 ? (1u << valid) - 1u : 0xFFFFFFFFu) : 0u;
        const uint32_t rows = b.y1 - b.y0, total = rows * (b.z1 - b.z0);
        for (uint32_t j = threadIdx.x; j < total; j += 256)
            A.g.bits[((uint64_t)(b.z0 + j / rows) * A.g.ny + b.y0 + j % rows) * A.g.W + b.wx] = word;
        if (threadIdx.x == 0) A.len[box] = 0;
        return;
    }
    // the last reset of the range, and the lowest ub from there on (or of the whole range)
    uint32_t reset = 0xFFFFFFFFu;
    float since = INF;
    each([&](uint32_t t, float d) {
        const uint32_t i = i0 + 32 * t;
        const float lb = d - spread, ub = d + spread;
        const float li = warp_incl_min(lb, lane);
        float le = __shfl_up_sync(0xFFFFFFFFu, li, 1);
        le = lane ? fminf(le, low) : low;
        low = fminf(low, __shfl_sync(0xFFFFFFFFu, li, 31));
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, i < A.n && ub + 2.0f * A.kpad <= le);
        uint32_t first = 0;
        if (m) {
            first = 31u - (uint32_t)__clz((int)m);
            reset = i - lane + first;
            since = INF;
        }
        if (lane >= first) since = fminf(since, ub);
    });
    for (int o = 16; o > 0; o >>= 1) since = fminf(since, __shfl_xor_sync(0xFFFFFFFFu, since, o));
    if (lane == 0) {
        s_reset[warp] = reset;
        s_since[warp] = since;
    }
    __syncthreads();
    uint32_t start_warp = 0;  // sphere 0 is always a reset
    for (uint32_t w = 0; w < 8; ++w)
        if (s_reset[w] != 0xFFFFFFFFu) start_warp = w;
    const uint32_t start = s_reset[start_warp];
    float up = INF;
    for (uint32_t w = start_warp; w < warp; ++w) up = fminf(up, s_since[w]);
    uint32_t cnt = 0;
    if (warp >= start_warp) {
        each([&](uint32_t t, float held_d) {
            const uint32_t i = i0 + 32 * t;
            const float d = i >= start ? held_d : INF, lb = d - spread, ub = d + spread;
            const float ui = warp_incl_min(ub, lane);
            float ue = __shfl_up_sync(0xFFFFFFFFu, ui, 1);
            ue = lane ? fminf(ue, up) : up;
            up = fminf(up, __shfl_sync(0xFFFFFFFFu, ui, 31));
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, i < A.n && i >= start && lb < ue + A.kpad);
            if (lane == 0) s_keep[warp][t] = m;
            cnt += __popc(m);
        });
    }
    if (lane == 0) s_cnt[warp] = cnt;
    __syncthreads();
    uint32_t at = 0, total = 0;
    for (uint32_t w = 0; w < 8; ++w) {
        if (w < warp) at += s_cnt[w];
        total += s_cnt[w];
    }
    if (threadIdx.x == 0) A.len[box] = total <= A.cap ? total : SMOOTH_ALL;
    if (total > A.cap || warp < start_warp) return;
    uint16_t* list = A.list + (size_t)box * A.cap;
    for (uint32_t t = 0; t < steps; ++t) {
        const uint32_t m = s_keep[warp][t];
        if ((m >> lane) & 1u) list[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(i0 + 32 * t);
        at += __popc(m);
    }
}

// One block of 64 threads per box, thread = sub-brick (x fastest).
template <bool RK>
__global__ void __launch_bounds__(64) smooth_classify(SmoothArgs A) {
    const float INF = __int_as_float(0x7F800000);
    __shared__ float4 s_sp[64];
    __shared__ uint8_t s_cls[64];
    const uint32_t box = blockIdx.x, len = A.len[box];
    if (len == 0) return;
    const BrickLattice& g = A.g;
    const SmoothBox b = smooth_box(A, box);
    const bool all = len == SMOOTH_ALL;
    const uint32_t n = all ? A.n : len;
    const uint16_t* list = A.list + (size_t)box * A.cap;
    const uint32_t t = threadIdx.x, sy = A.rows / 4;  // sub-bricks along y and z
    const uint32_t xa = 32 * b.wx + 8 * (t & 3), ya = b.y0 + 4 * ((t >> 2) % sy), za = b.z0 + 4 * ((t >> 2) / sy);
    const bool live = t < A.nsub && xa < g.nx && ya < b.y1 && za < b.z1;
    V3 c = v3(0.0f, 0.0f, 0.0f);
    float spread = 0.0f;
    if (live)
        spread = smooth_spread(A, xa, min(xa + 7, g.nx - 1), ya, min(ya + 3, b.y1 - 1), za, min(za + 3, b.z1 - 1), &c);
    // the fold at the centre; the partial fold too changes by at most spread
    // over the sub-brick, so it bounds itself there
    float v = INF;
    uint32_t first = 0, word = 0;
    uint32_t* mask = A.mask + (size_t)box * (A.cap / 32) * A.nsub + t;
    for (uint32_t p0 = 0; p0 < n; p0 += 64) {
        __syncthreads();  // the previous spheres are used
        if (p0 + t < n) s_sp[t] = __ldg(A.sp + (all ? p0 + t : (uint32_t)list[p0 + t]));
        __syncthreads();
        if (!live) continue;
        const uint32_t m = min(64u, n - p0);
        for (uint32_t j = 0; j < m; ++j) {
            const float4 s = s_sp[j];
            // d - spread >= v + spread + k leaves v as it is: decided from the
            // squared distance, without the root, for most of the spheres
            const float sq = len_sq(v3(c.x - s.x, c.y - s.y, c.z - s.z)), e = v + (2.0f * spread + A.kpad + s.w);
            if (e > 0.0f && sq < e * e) {
                const float d = sqrtf(sq) - s.w;
                word |= 1u << (j & 31);
                if (d + spread + A.kpad <= v - spread) {  // reset
                    first = p0 + j;
                    v = d;
                } else {
                    v = smooth_min_by<RK>(v, d, A.k, A.rk);
                }
            }
            if ((j & 31) == 31 || j + 1 == m) {
                if (!all) mask[(size_t)((p0 + j) / 32) * A.nsub] = word;
                word = 0;
            }
        }
    }
    const float reach = smooth_reach(g);
    uint32_t cls = BRICK_OUT;
    if (live) cls = v - spread > reach ? BRICK_OUT : (v + spread < -reach ? BRICK_IN : BRICK_MIXED);
    s_cls[t] = (uint8_t)cls;
    const bool mixed = live && cls == BRICK_MIXED;
    const uint32_t lane = t & 31, m = __ballot_sync(0xFFFFFFFFu, mixed);
    if (m) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(A.ntasks, (uint32_t)__popc(m));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (mixed) A.tasks[base + __popc(m & ((1u << lane) - 1u))] = make_uint2(box * A.nsub + t, first);
    }
    __syncthreads();
    // sign bits: thread = (row of the box, layer in steps), one word per row;
    // smooth_rows writes the mixed sub-bricks' bytes after this
    for (uint32_t r = t; r < A.rows * A.rows; r += 64) {
        const uint32_t yr = r % A.rows, zr = r / A.rows, y = b.y0 + yr, z = b.z0 + zr;
        if (y >= b.y1 || z >= b.z1) continue;
        uint32_t cls4 = 0;
        for (uint32_t j = 0; j < 4; ++j) cls4 |= (uint32_t)s_cls[((zr >> 2) * sy + (yr >> 2)) * 4 + j] << (8 * j);
        g.bits[((uint64_t)z * g.ny + y) * g.W + b.wx] = decided_word(cls4, g.nx, b.wx);
    }
}

// A warp per mixed sub-brick over a persistent grid, four samples per lane:
// the 32 lanes are 4 x 4 x 2 neighbouring samples (as compact as 32 samples
// get, so that they need the same spheres), the four samples of a lane the
// sub-brick's halves along x and z.  32 list positions at a time are gathered
// to shared memory and the kept ones folded in order.
template <bool RK>
__global__ void __launch_bounds__(256) smooth_rows(SmoothArgs A) {
    const float INF = __int_as_float(0x7F800000);
    __shared__ float4 s_sp[8][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const BrickLattice& g = A.g;
    const uint32_t ntasks = *A.ntasks;
    for (uint32_t q = blockIdx.x * 8 + warp; q < ntasks; q += gridDim.x * 8) {
        const uint2 task = A.tasks[q];
        const uint32_t box = task.x / A.nsub, t = task.x % A.nsub;
        const SmoothBox b = smooth_box(A, box);
        const uint32_t len = A.len[box];
        const bool all = len == SMOOTH_ALL;
        const uint32_t n = all ? A.n : len, sy = A.rows / 4;
        const uint32_t x0 = 32 * b.wx + 8 * (t & 3), y0 = b.y0 + 4 * ((t >> 2) % sy), z0 = b.z0 + 4 * ((t >> 2) / sy);
        const uint32_t x = x0 + (lane & 3), y = y0 + ((lane >> 2) & 3), z = z0 + (lane >> 4);
        const uint16_t* list = A.list + (size_t)box * A.cap;
        const uint32_t* mask = A.mask + (size_t)box * (A.cap / 32) * A.nsub + t;
        const V3 p = smooth_point(A, v3((float)x * g.inv, (float)y * g.inv, (float)(z + g.zoff) * g.inv));
        const V3 r = smooth_point(A, v3((float)(x + 4) * g.inv, (float)y * g.inv, (float)(z + 2 + g.zoff) * g.inv));
        // from +infinity the first sphere replaces the value, as the fold's start does
        float v[4] = {INF, INF, INF, INF};
        for (uint32_t w = task.y / 32; 32 * w < n; ++w) {
            uint32_t m = all ? 0xFFFFFFFFu : __ldg(mask + (size_t)w * A.nsub);
            if (32 * w < task.y) m &= ~0u << (task.y & 31);
            if (n - 32 * w < 32) m &= (1u << (n - 32 * w)) - 1u;
            if (!m) continue;
            __syncwarp();  // the previous spheres are used
            if ((m >> lane) & 1u) {
                const uint32_t i = 32 * w + lane;
                s_sp[warp][__popc(m & ((1u << lane) - 1u))] = __ldg(A.sp + (all ? i : (uint32_t)__ldg(list + i)));
            }
            __syncwarp();
            const uint32_t cnt = __popc(m);
            for (uint32_t j = 0; j < cnt; ++j) {
                const float4 s = s_sp[warp][j];
                const float dy = p.y - s.y, dyy = dy * dy;
                const float dx0 = p.x - s.x, dx1 = r.x - s.x, dz0 = p.z - s.z, dz1 = r.z - s.z;
                const float xy[2] = {dx0 * dx0 + dyy, dx1 * dx1 + dyy}, zz[2] = {dz0 * dz0, dz1 * dz1};
                const float pad = s.w + A.kpad;
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    // d >= v + k leaves v as it is: decided from the squared
                    // distance, without the root, for most of the spheres
                    const float sq = xy[l & 1] + zz[l >> 1], e = v[l] + pad;
                    if (e > 0.0f && sq < e * e) v[l] = smooth_min_by<RK>(v[l], sqrtf(sq) - s.w, A.k, A.rk);
                }
            }
        }
        uint32_t bits[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const uint32_t xl = x + 4 * (l & 1), zl = z + 2 * (l >> 1);
            const bool ok = y < b.y1 && zl < b.z1 && xl < g.nx;
            if (ok) g.field[((uint64_t)zl * g.ny + y) * g.pitch + xl] = v[l];
            bits[l] = __ballot_sync(0xFFFFFFFFu, ok && !(v[l] > 0.0f));
        }
        // lanes 0-15: one row's sign byte each, from its two half rows
        const uint32_t yr = lane & 3, zr = (lane >> 2) & 3;
        if (lane < 16 && y0 + yr < b.y1 && z0 + zr < b.z1) {
            const uint32_t sh = 4 * yr + 16 * (zr & 1);
            const uint32_t lo = ((zr & 2) ? bits[2] : bits[0]) >> sh, hi = ((zr & 2) ? bits[3] : bits[1]) >> sh;
            reinterpret_cast<uint8_t*>(g.bits + ((uint64_t)(z0 + zr) * g.ny + y0 + yr) * g.W + b.wx)[t & 3] =
                (uint8_t)((lo & 15u) | (hi & 15u) << 4);
        }
    }
}

}  // namespace

// Whether the extractors' samples of this program take the culled smooth
// union.  Below 16 spheres a box list saves nothing over the general culled
// sampler; without a Lipschitz bound there is nothing to cull by; beyond
// magnitudes of about 10^13 squared distances near f32's range, where the
// bounds above would no longer be finite.  (The slack is 2^-13 of the largest
// magnitude, the width's included, so this also ends the widths, near 2^43.)
static bool smooth_culled(const iso_program* prog, uint32_t nx, uint32_t ny, uint32_t nz) {
    return prog->smooth_set && prog->lip > 0.0f && prog->slack < 1e9f && prog->set_n >= 16 && prog->set_n <= SMOOTH_MAX && nx > 1 &&
           (uint64_t)words_per_row(nx) * ((ny + 3) / 4) * ((nz + 3) / 4) < (1ull << 26);
}

static iso_status launch_smooth_set(iso_ctx* ctx, const iso_program* prog, const BrickLattice& g) {
    SmoothArgs A{};
    A.sp = (const float4*)prog->d_set;
    A.n = prog->set_n;
    A.k = prog->set_k;
    A.kpad = prog->set_k * (1.0f + 1.0f / 1024.0f) + prog->slack;
    A.rk = A.k >= 0x1p-60f ? 1.0f / A.k : 0.0f;  // (smooth_culled ends the widths far below 2^60)
    A.domain = prog->has_domain;
    A.sx = prog->domain[0]; A.sy = prog->domain[1]; A.sz = prog->domain[2];
    A.ox = prog->domain[3]; A.oy = prog->domain[4]; A.oz = prog->domain[5];
    A.g = g;
    // boxes of 16 rows and layers; smaller ones while a small lattice would
    // leave SMs without a box
    A.rows = 16;
    auto boxes = [&](uint32_t rows) { return (uint64_t)g.W * ((g.ny + rows - 1) / rows) * ((g.nz + rows - 1) / rows); };
    while (A.rows > 4 && boxes(A.rows) < 8ull * (uint64_t)ctx->sms) A.rows /= 2;
    A.by = (g.ny + A.rows - 1) / A.rows;
    A.bz = (g.nz + A.rows - 1) / A.rows;
    A.nsub = A.rows * A.rows / 4;
    const uint64_t nb = boxes(A.rows);
    // list room per box: every sphere while the lists and masks stay within
    // 160 MB (many boxes are small ones with short lists), at least 512
    const uint64_t per_entry = 2 + A.nsub / 8;
    const uint64_t all = ((uint64_t)A.n + 31) & ~31ull;
    A.cap = (uint32_t)std::min<uint64_t>(all, std::max<uint64_t>(512, (160ull << 20) / (nb * per_entry) & ~31ull));
    auto at256 = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t o_len = 256, o_list = at256(o_len + 4 * nb), o_mask = at256(o_list + 2 * nb * A.cap);
    const size_t o_tasks = at256(o_mask + nb * A.nsub * (A.cap / 8));
    iso_status s = ensure(ctx, ctx->tiles, o_tasks + 8 * nb * A.nsub);
    if (s != ISO_OK) return s;
    char* base = (char*)ctx->tiles.p;
    A.ntasks = (uint32_t*)base;
    A.len = (uint32_t*)(base + o_len);
    A.list = (uint16_t*)(base + o_list);
    A.mask = (uint32_t*)(base + o_mask);
    A.tasks = (uint2*)(base + o_tasks);
    cudaError_t e = cudaMemsetAsync(A.ntasks, 0, 4, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "smooth set task count");
    StageTimer timer(ctx, ISO_STAGE_SAMPLE);
    smooth_boxes<<<(unsigned)nb, 256, 0, ctx->stream>>>(A);
    if (A.rk != 0.0f) smooth_classify<true><<<(unsigned)nb, 64, 0, ctx->stream>>>(A);
    else smooth_classify<false><<<(unsigned)nb, 64, 0, ctx->stream>>>(A);
    auto* const rows = A.rk != 0.0f ? smooth_rows<true> : smooth_rows<false>;
    rows<<<persistent_blocks(ctx, (const void*)rows), 256, 0, ctx->stream>>>(A);
    ctx->launches += 2;
    return ISO_OK;
}

}  // namespace iso
