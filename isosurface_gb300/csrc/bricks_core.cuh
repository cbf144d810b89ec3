// Culled sampling of a general program for marching cubes (and, at the end,
// the plain sampler of every point): the device code, written so that it
// also compiles on its own under NVRTC (no includes: the
// library includes it after its own headers, the run-time compiler after a
// prelude of fixed-width integer types and vm_math.cuh).
//
// Marching cubes reads a sample's value only at the ends of crossing edges
// (sign change between lattice neighbours one step `inv` apart), and both
// ends of such an edge lie within lip * inv of zero when the program's value
// is lip-Lipschitz in the sample point.  A sub-brick of 8 (x) x 4 (y) x 4 (z)
// points whose centre value v satisfies |v| > lip * h + lip * inv (h: the
// distance from the centre to its farthest point; plus rounding slack) holds
// no such end: all its samples have v's sign and no value of it is ever
// read.  Such a sub-brick gets sign bits only; every sample of the others is
// evaluated with the program's evaluator, so every value written is
// bit-identical to the full sampler's, and so is every sign bit.
//
// For a hard union of translated primitives (at most 64) each sub-brick also
// keeps only the primitives that can attain the minimum in it: primitive i's
// values over the sub-brick lie within lip * h of d_i(centre), so i is
// dropped when d_i - lip * h exceeds min_j (d_j + lip * h); the minimum over
// the kept ones equals the minimum over all.
//
// Work is cut in tiles: all x, rows [y0, y1), layers [z0, z1), y0 and z0
// multiples of 4, at most BRICK_MAX sub-bricks.  One thread classifies one
// sub-brick.  A group of four sub-bricks along x (32 x 4 x 4 points, one
// sign word in each of 16 rows) that is wholly decided gets its sign words
// at once; in a mixed group every sample of the mixed ones is evaluated
// afterwards, four mixed sub-bricks to a warp (eight lanes each, one sign byte
// per row), so that no lane idles on a decided sub-brick.  Classification
// appends the mixed sub-bricks to a list (a block per tile here; a warp per 32
// sub-bricks for many small lattices, batch.cu); a persistent grid then
// samples the list, so the evaluation is spread evenly however the surface
// falls.
//
// The evaluator `Ev` provides value(p) and, for pruned unions, prunable(),
// nprims(), point(p) (the point after a leading domain map, which keeps the
// axes apart), prim(i, q) and values_kept(keep, p, v): v[4 k + j] is the
// union's value at (p[0].x, p[j].y, p[k].z).
#pragma once

namespace iso {

constexpr uint32_t BRICK_MAX = 1024;        // sub-bricks per tile
constexpr uint32_t BRICK_PRUNE_MAX = 64;    // primitives a keep mask covers
constexpr uint32_t BRICK_ERR_CAPACITY = 2u;  // error bit: a list ran out of room
enum : uint32_t { BRICK_MIXED = 0, BRICK_OUT = 1, BRICK_IN = 2 };

struct BrickLattice {
    float lip;    // Lipschitz bound of the program's value in the sample point
    float slack;  // rounding slack of two values the evaluator computes
    uint32_t nx, ny, nz;  // samples per axis
    float inv;            // lattice step in sample coordinates
    float* field;
    uint64_t pitch;
    uint32_t* bits;
    uint32_t W;     // sign words per row
    uint32_t zoff;  // lattice z of layer 0 (a slab of a larger lattice)
    float reach_steps;  // values are needed within this many lattice steps' worth of change of zero
};

// One tile: the lattice and its rows / layers.
struct BrickTile {
    BrickLattice g;
    uint32_t y0, y1, z0, z1;
};

// A mixed sub-brick: tile * BRICK_MAX + sub-brick, and the primitives it keeps.
struct BrickTask {
    uint32_t tile_sb, unused;
    uint64_t keep;
};

// The tiles of one lattice: 4 layers x `rows` rows each.
struct GridTiles {
    BrickLattice g;
    uint32_t rows, ytiles;
    __device__ __forceinline__ BrickTile tile(uint32_t t) const {
        const uint32_t y0 = (t % ytiles) * rows, z0 = 4 * (t / ytiles);
        return BrickTile{g, y0, min(y0 + rows, g.ny), z0, min(z0 + 4, g.nz)};
    }
};

// OR of a 64-bit mask over the warp (every lane calls it).
__device__ __forceinline__ uint64_t warp_or64(uint64_t m) {
    const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)m);
    const uint32_t hi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(m >> 32));
    return ((uint64_t)hi << 32) | lo;
}

// Sub-bricks of a tile covering `rows` rows and `layers` layers.
__host__ __device__ __forceinline__ uint32_t brick_count(uint32_t W, uint32_t rows, uint32_t layers) {
    return 4 * W * ((rows + 3) / 4) * ((layers + 3) / 4);
}

// Class of the sub-brick of samples [xa, xb] x [ya, yb] x [za, zb] and the
// primitives it keeps (a program with a bound).  The values of the first
// `nheld` primitives are held at held[0], held[stride], ... for the second
// look at them (null: all are evaluated twice).
template <class Ev>
__device__ __forceinline__ uint32_t brick_class(const Ev& ev, const BrickLattice& g, uint32_t xa, uint32_t xb,
                                                uint32_t ya, uint32_t yb, uint32_t za, uint32_t zb, uint64_t* keep,
                                                float* held = nullptr, uint32_t nheld = 0, uint32_t stride = 0) {
    // both ends of a crossing edge lie within lip * inv of zero (rounded up);
    // a caller may need values further out (reach_steps > 1)
    const float reach = g.lip * g.inv * g.reach_steps * (1.0f + 1.0f / 1024.0f) + g.slack;
    const float hx = 0.5f * (float)(xb - xa), hy = 0.5f * (float)(yb - ya), hz = 0.5f * (float)(zb - za);
    const V3 c = v3(((float)xa + hx) * g.inv, ((float)ya + hy) * g.inv, ((float)(za + g.zoff) + hz) * g.inv);
    // the largest change of any value over the sub-brick, rounded up
    const float spread = g.lip * sqrtf((hx * hx + hy * hy) + hz * hz) * g.inv * (1.0f + 1.0f / 1024.0f) + g.slack;
    float v;
    if (ev.prunable()) {
        const V3 q = ev.point(c);
        const uint32_t n = ev.nprims();
        float upper = __int_as_float(0x7F800000);  // +infinity
        v = 0.0f;
        for (uint32_t i = 0; i < n; ++i) {
            const float d = ev.prim(i, q);
            v = (i == 0) ? d : fminf(v, d);
            upper = fminf(upper, d + spread);
            if (i < nheld) held[i * stride] = d;
        }
        uint64_t k = 0;
        for (uint32_t i = 0; i < n; ++i) {
            const float d = i < nheld ? held[i * stride] : ev.prim(i, q);
            if (!(d - spread > upper)) k |= 1ull << i;
        }
        *keep = k;
    } else {
        v = ev.value(c);
    }
    if (v - spread > reach) return BRICK_OUT;
    if (v + spread < -reach) return BRICK_IN;
    return BRICK_MIXED;
}

// Class and kept primitives of every sub-brick of a tile, into shared memory
// (every thread of the block calls it; no barrier at the end).
template <class Ev>
__device__ __forceinline__ void brick_classes(const Ev& ev, const BrickTile& T, uint8_t* s_cls, uint64_t* s_keep) {
    const BrickLattice& g = T.g;
    const uint32_t SX = 4 * g.W, SY = (T.y1 - T.y0 + 3) / 4, SZ = (T.z1 - T.z0 + 3) / 4;
    const uint32_t nsb = SX * SY * SZ;
    for (uint32_t s = threadIdx.x; s < nsb; s += blockDim.x) {
        uint32_t cls = BRICK_MIXED;
        uint64_t keep = ~0ull;
        if (g.lip > 0.0f) {
            const uint32_t sx = s % SX, sy = (s / SX) % SY, sz = s / (SX * SY);
            const uint32_t xa = 8 * sx, ya = T.y0 + 4 * sy, za = T.z0 + 4 * sz;
            if (xa >= g.nx) cls = BRICK_OUT;  // no samples: sign bits stay clear
            else
                cls = brick_class(ev, g, xa, min(xa + 7, g.nx - 1), ya, min(ya + 3, T.y1 - 1), za,
                                  min(za + 3, T.z1 - 1), &keep);
        }
        s_cls[s] = (uint8_t)cls;
        s_keep[s] = keep;
    }
}

// Sign word of a group from its sub-bricks' classes, bits of mixed ones and
// past the row's last sample clear.
__device__ __forceinline__ uint32_t decided_word(uint32_t cls4, uint32_t nx, uint32_t w) {
    uint32_t word = 0;
    for (uint32_t j = 0; j < 4; ++j)
        if (((cls4 >> (8 * j)) & 0xFFu) == BRICK_IN) word |= 0xFFu << (8 * j);
    const uint32_t valid = nx - 32 * w;  // samples of this word (> 0)
    return valid < 32 ? word & ((1u << valid) - 1u) : word;
}

// The sign bits of group gi of tile T (four sub-bricks along x, one sign
// word in each of 16 rows), written by one thread; brick_quad writes the
// bytes of the mixed sub-bricks after that (writing only the decided ones'
// here took up to 64 byte stores).  Returns the mask of mixed sub-bricks (bit
// j: sub-brick 4 gi + j).
__device__ __forceinline__ uint32_t brick_group_bits(const BrickTile& T, uint32_t gi, const uint8_t* s_cls) {
    const BrickLattice& g = T.g;
    const uint32_t SY = (T.y1 - T.y0 + 3) / 4;
    const uint32_t w = gi % g.W, gy = (gi / g.W) % SY, gz = gi / (g.W * SY);
    uint32_t cls4 = 0, mixed = 0;
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t c = s_cls[4 * gi + j];
        cls4 |= c << (8 * j);
        if (c == BRICK_MIXED) mixed |= 1u << j;
    }
    const uint32_t word = decided_word(cls4, g.nx, w);
    for (uint32_t r = 0; r < 16; ++r) {
        const uint32_t y = T.y0 + 4 * gy + (r & 3), z = T.z0 + 4 * gz + (r >> 2);
        if (y >= T.y1 || z >= T.z1) continue;
        g.bits[((uint64_t)z * g.ny + y) * g.W + w] = word;
    }
    return mixed;
}

// The 16 rows of up to four mixed sub-bricks, one per eight lanes (sx, ya,
// za and have: the lane's own sub-brick; y1, z1: the ends of its rows): lane
// l samples x = 8 sx + l % 8, and the eight lanes' signs go out as one byte
// of the row's sign word.  `keep` (the same in every lane) holds every
// primitive any of the sub-bricks keeps.  Every lane of the warp calls it.
//
// A pruned union is evaluated a primitive at a time over the lane's 4 x 4
// points (values_kept): the primitive is read and told apart once for 16
// points, and what depends on one or two of the coordinates is computed
// once per coordinate.  The chunk batch's 1024 chunks: 109 M warp
// instructions for the mixed sub-bricks, 348 M with a point at a time
// (classification included).
template <class Ev>
__device__ __forceinline__ void brick_fill(const Ev& ev, const BrickLattice& g, bool have, uint32_t sx, uint32_t ya,
                                           uint32_t za, uint32_t y1, uint32_t z1, uint64_t keep) {
    const uint32_t lane = threadIdx.x & 31, x = 8 * sx + (lane & 7);
    auto put = [&](uint32_t r, float v) {
        const uint32_t y = ya + (r & 3), z = za + (r >> 2);
        const bool row_ok = have && y < y1 && z < z1;
        const uint64_t row = (uint64_t)z * g.ny + y;
        const bool in = row_ok && x < g.nx;
        if (in) g.field[row * g.pitch + x] = v;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, in && !(v > 0.0f));
        if (row_ok && (lane & 7) == 0)
            reinterpret_cast<uint8_t*>(g.bits + row * g.W + sx / 4)[sx % 4] = (uint8_t)(b >> (lane & ~7u));
    };
    if (g.lip > 0.0f && ev.prunable()) {
        V3 p[4];  // (x, y_j, z_j)
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            p[j] = v3((float)x * g.inv, (float)(ya + j) * g.inv, (float)(za + j + g.zoff) * g.inv);
        float v[16];
        ev.values_kept(keep, p, v);
#pragma unroll
        for (uint32_t r = 0; r < 16; ++r) put(r, v[r]);
        return;
    }
    for (uint32_t r = 0; r < 16; ++r) {
        const uint32_t y = ya + (r & 3), z = za + (r >> 2);
        float v = 0.0f;
        if (have && y < y1 && z < z1 && x < g.nx)
            v = ev.value(v3((float)x * g.inv, (float)y * g.inv, (float)(z + g.zoff) * g.inv));
        put(r, v);
    }
}

// brick_fill of sub-brick `sb` of tile `T` (the lane's own; sb = ~0u: none)
template <class Ev>
__device__ __forceinline__ void brick_quad(const Ev& ev, const BrickTile& T, uint32_t sb, uint64_t keep) {
    const BrickLattice& g = T.g;
    const uint32_t lane = threadIdx.x & 31;
    const bool have = sb != 0xFFFFFFFFu;
    uint32_t sx = 0, ya = 0, za = 0;
    if (have) {
        const uint32_t SX = 4 * g.W, SY = (T.y1 - T.y0 + 3) / 4;
        sx = sb % SX;
        ya = T.y0 + 4 * ((sb / SX) % SY);
        za = T.z0 + 4 * (sb / (SX * SY));
    }
    brick_fill(ev, g, have, sx, ya, za, T.y1, T.z1, keep);
}

// Classify one tile, write its decided sign bits and list its mixed
// sub-bricks (every thread of the block calls it).
template <class Ev>
__device__ __forceinline__ void brick_classify_tile(const Ev& ev, const BrickTile& T, uint32_t tile, uint8_t* s_cls,
                                                    uint64_t* s_keep, BrickTask* list, uint32_t* count,
                                                    uint32_t cap, uint32_t* err) {
    brick_classes(ev, T, s_cls, s_keep);
    __syncthreads();
    const uint32_t groups = brick_count(T.g.W, T.y1 - T.y0, T.z1 - T.z0) / 4, lane = threadIdx.x & 31;
    for (uint32_t gb = 0; gb < groups; gb += blockDim.x) {
        const uint32_t gi = gb + threadIdx.x;
        const uint32_t mixed = gi < groups ? brick_group_bits(T, gi, s_cls) : 0u;
        // warp-aggregated append of the mixed sub-bricks
        const uint32_t n = __popc(mixed);
        uint32_t incl = n;
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += o;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (total) {
            uint32_t base = 0;
            if (lane == 31) base = atomicAdd(count, total);
            base = __shfl_sync(0xFFFFFFFFu, base, 31) + incl - n;
            for (uint32_t m = mixed; m; m &= m - 1, ++base) {
                const uint32_t sb = 4 * gi + (uint32_t)(__ffs(m) - 1);
                if (base < cap) list[base] = BrickTask{tile * BRICK_MAX + sb, 0, s_keep[sb]};
                else atomicOr(err, BRICK_ERR_CAPACITY);
            }
        }
    }
}

// The bodies of the two single-lattice kernels (Tiles: a type with
// `BrickTile tile(uint32_t) const` on the device; blocks of 256 threads).
template <class Tiles, class Ev>
__device__ __forceinline__ void brick_classify_body(const Ev& ev, const Tiles& tiles, BrickTask* list,
                                                    uint32_t* count, uint32_t cap, uint32_t* err) {
    __shared__ uint8_t s_cls[BRICK_MAX];
    __shared__ uint64_t s_keep[BRICK_MAX];
    brick_classify_tile(ev, tiles.tile(blockIdx.x), blockIdx.x, s_cls, s_keep, list, count, cap, err);
}

// The listed mixed sub-bricks, four to a warp, over a persistent grid.
template <class Tiles, class Ev>
__device__ __forceinline__ void brick_rows_body(const Ev& ev, const Tiles& tiles, const BrickTask* list,
                                                const uint32_t* count, uint32_t cap) {
    const uint32_t n = min(*count, cap), lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t q = 4 * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); q < n; q += 4 * warps) {
        const uint32_t e = q + (lane >> 3);
        BrickTask k{0, 0, 0};
        if (e < n) k = list[e];
        const uint64_t keep = warp_or64(k.keep);
        brick_quad(ev, tiles.tile(k.tile_sb / BRICK_MAX), e < n ? k.tile_sb % BRICK_MAX : 0xFFFFFFFFu, keep);
    }
}

// The plain sampler (every point, nothing culled; the lattice's culling
// fields unused): warp gw of the lattice's W * ny * nz takes 32 consecutive
// points of one row, writes their values and, by ballot, the row's sign word.
template <class Ev>
__device__ __forceinline__ void field_warp(const Ev& ev, const BrickLattice& g, uint64_t gw) {
    if (gw >= (uint64_t)g.W * g.ny * g.nz) return;  // warp-uniform
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t w = (uint32_t)(gw % g.W);
    const uint64_t row = gw / g.W;
    const uint32_t y = (uint32_t)(row % g.ny), z = (uint32_t)(row / g.ny);
    const uint32_t x = 32 * w + lane;
    bool inside = false;
    if (x < g.nx) {
        const float v = ev.value(v3((float)x * g.inv, (float)y * g.inv, (float)(z + g.zoff) * g.inv));
        g.field[row * g.pitch + x] = v;
        inside = !(v > 0.0f);
    }
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, inside);
    if (lane == 0) g.bits[row * g.W + w] = b;
}

}  // namespace iso
