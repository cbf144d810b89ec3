// The cell passes of marching cubes (included by mc.cu inside
// iso::{anonymous}, after mc_chunk.cuh): one lattice, or a table of lattices
// whose edge maps share one 32-bit key space.
//
// A segment is 32 consecutive chunks of one cell layer in (y, x) order (a
// chunk is 32 cells of a row; a layer's last segment may be shorter), or
// eight in small lattices and tables, so segments in order are the
// reference's (z, y, x) visit order.  A counting warp handles 32 chunks with
// lane = chunk.
//
//   mc_cell_count   owned vertices and triangles of every segment, from the
//                   sign bits
//   mc_cell_scan    exclusive prefixes, and the list of the segments that
//                   hold any active cell
//   mc_cell_emit    vertices, the edge map and triangles (as map keys) of the
//                   listed segments
//   mc_resolve_ids  keys -> vertex ids
//
// 513^3 samples of a 64-sphere union (4.2 M chunks, 1.5 M active cells), one
// kernel after the other: count 28 us (bound by its ALU pipe, 70 %), scan 8,
// emit 69 (issue and load latency: 57 % of the slots while busy; dense
// segments finish last).  The passes they replace, which loaded every
// chunk's eight words in each of two kernels and looked every active cell's
// triangle count up: count and scan 55, emit 79.  401 x 401 x 301 samples of
// a dense field: 18 + 8 + 114 against 48 + 126.  A dual lattice of 256^3: 9 +
// 8 + 28 against 19 + 4 + 50 with the block emit.  A table of 1024 lattices
// of 16^3 to 64^3 cells: 25 + 9 + 116 and 46 for the ids against 55 + 9 + 305
// with the block emit.
constexpr uint32_t SCAN_BLOCK_SEGS = 4096;  // segments per block of mc_cell_scan (512 threads x 8)

struct CellArgs {
    Grid grid;           // one lattice
    const Grid* grids;   // or a table
    const uint32_t* seg_grid;  // table: the lattice of each segment
    const uint4* tasks;  // table: mc_cell_count's tasks (lattice, segment of the layer, first layer, layers)
    uint32_t ntasks;     // mc_cell_count: warps with work
    uint32_t run;        // one lattice: layers per task
    uint32_t nsegs;
    uint2* segs;         // per segment: (vertices, triangles), then their prefix inside its scan block
    uint32_t* masks;     // per segment: its active chunks
    uint2* blocks;       // per scan block: totals
    uint32_t nblocks;
    uint32_t group;      // list entries an emitting warp takes together
    uint4* list;         // active segments: (segment, vertex prefix, triangle prefix, active chunks)
    uint32_t* ctrl;      // [0] length of the list [1] groups taken from it beyond each emitting warp's first
    uint64_t* totals;    // [0] triangles [1] vertices
    uint32_t* err;
};

// ---------------------------------------------------------------- counting ---
// The four sign rows' words around a chunk, of one sample layer: corners 0-3
// (or 4-7, a layer up) of its 32 cells.
struct Quad {
    uint32_t k[4];
};

__device__ __forceinline__ Quad load_quad(const uint32_t* __restrict__ p, uint32_t W, bool in, bool nxt) {
    const uint32_t a0 = in ? __ldg(p) : 0u, an = nxt ? __ldg(p + 1) : 0u;
    const uint32_t b0 = in ? __ldg(p + W) : 0u, bn = nxt ? __ldg(p + W + 1) : 0u;
    // CORNERS order: (x,y) (x+1,y) (x+1,y+1) (x,y+1)
    return Quad{{a0, __funnelshift_r(a0, an, 1), __funnelshift_r(b0, bn, 1), b0}};
}

__device__ __forceinline__ uint32_t maj(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (c & (a | b)); }

// A warp marches its 32 chunks up `run` layers, the sign words of a layer
// serving the cells below and above it, so a step costs four loads (the next
// layer's are in flight meanwhile) and, without an active cell, a handful of
// bit operations.  Every counted quantity comes from bit vectors: a case with
// e crossing edges has e - 2 triangles per loop of edges (checked against
// the tables when they are generated), only cases with six or more have a
// second loop, and e summed over the chunk comes from bit-sliced adders; the
// few cells with six or more look their case up.
template <bool TABLE, uint32_t SHIFT>
__global__ void __launch_bounds__(256) mc_cell_count(CellArgs A) {
    __shared__ uint8_t s_extra[256];  // per case: loops after the first
    __shared__ uint16_t s_owned[8];
    const uint32_t lane = threadIdx.x & 31;
    {
        const uint32_t e = iso_edge_count[threadIdx.x], t = iso_tri_count[threadIdx.x];
        s_extra[threadIdx.x] = (uint8_t)(t ? (e - 2 - t) / 2 : 0);
    }
    if (threadIdx.x < 8) s_owned[threadIdx.x] = iso_owned_mask[threadIdx.x];
    __syncthreads();
    pdl_wait();     // the sign bits; the previous extraction's use of the control words
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x < 2) A.ctrl[threadIdx.x] = 0;
    const uint32_t task = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (task >= A.ntasks) return;
    uint4 t;
    if (TABLE) {
        t = __ldg(A.tasks + task);
    } else {
        const uint32_t r = fdiv(task, A.grid.div_wl);
        t.y = task - r * A.grid.WL;
        t.z = r * A.run;
        t.w = min(A.run, A.grid.nz - 1 - t.z);
    }
    const Grid g = TABLE ? A.grids[t.x] : A.grid;
    const uint32_t l = 32 * t.y + lane, y = fdiv(l, g.div_cw), c = l - y * g.CW;
    const bool in = l < g.S, nxt = in && c + 1 < g.W;
    const uint32_t valid = in ? chunk_valid(c, g.nx - 1) : 0u;
    const uint64_t layer = (uint64_t)g.ny * g.W;
    const uint32_t* p = g.bits + t.z * layer + (uint64_t)y * g.W + c;
    // the lane's segment, and whether its first lane writes the counts
    constexpr uint32_t per = 1u << SHIFT;
    const uint32_t sl = l >> SHIFT, first = lane & ~(per - 1);
    const bool writes = lane == first && sl < g.SL;
    uint32_t seg = g.seg0 + t.z * g.SL + sl;
    Quad lo = load_quad(p, g.W, in, nxt);
    p += layer;
    Quad up = load_quad(p, g.W, in, nxt);
    uint32_t any_lo = lo.k[0] | lo.k[1] | lo.k[2] | lo.k[3], all_lo = lo.k[0] & lo.k[1] & lo.k[2] & lo.k[3];
    for (uint32_t i = 0; i < t.w; ++i, seg += g.SL) {
        const Quad hi = up;
        if (i + 1 < t.w) {
            p += layer;
            up = load_quad(p, g.W, in, nxt);
        }
        const uint32_t any_hi = hi.k[0] | hi.k[1] | hi.k[2] | hi.k[3], all_hi = hi.k[0] & hi.k[1] & hi.k[2] & hi.k[3];
        const uint32_t act = (any_lo | any_hi) & ~(all_lo & all_hi) & valid;
        uint32_t v = 0, tri = 0;
        const uint32_t chunks = __ballot_sync(FULL, act != 0);
        if (chunks) {
            const uint32_t z = t.z + i;
            const Corners q{{lo.k[0], lo.k[1], lo.k[2], lo.k[3], hi.k[0], hi.k[1], hi.k[2], hi.k[3]}};
            if (act) {
                if (y > 0 && z > 0) {
                    // interior row: cells own edges 5 (k5^k6), 6 (k6^k7), 10 (k2^k6);
                    // the row's x == 0 cell also owns 7 (k7^k4) and 11 (k3^k7)
                    v = __popc((q.k[5] ^ q.k[6]) & act) + __popc((q.k[6] ^ q.k[7]) & act) +
                        __popc((q.k[2] ^ q.k[6]) & act);
                    if (c == 0 && (act & 1u)) v += ((q.k[7] ^ q.k[4]) & 1u) + ((q.k[3] ^ q.k[7]) & 1u);
                } else {
                    const int cls = (y == 0 ? 2 : 0) | (z == 0 ? 4 : 0);
                    v = owned_count(q, act, s_owned[cls], s_owned[cls | 1], c == 0 ? 1u : 0u);
                }
                // crossing edges per cell, bit-sliced: s0 + 2 s1 + 4 s2 + 8 s3
                constexpr uint8_t EC[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                               {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
                uint32_t x[12];
#pragma unroll
                for (int e = 0; e < 12; ++e) x[e] = (q.k[EC[e][0]] ^ q.k[EC[e][1]]) & act;
                uint32_t one[4], two[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    one[j] = x[3 * j] ^ x[3 * j + 1] ^ x[3 * j + 2];
                    two[j] = maj(x[3 * j], x[3 * j + 1], x[3 * j + 2]);
                }
                const uint32_t o3 = one[0] ^ one[1] ^ one[2], t4 = maj(one[0], one[1], one[2]);
                const uint32_t s0 = o3 ^ one[3], t5 = o3 & one[3];
                const uint32_t u0 = two[0] ^ two[1] ^ two[2], f0 = maj(two[0], two[1], two[2]);
                const uint32_t u1 = two[3] ^ t4 ^ t5, f1 = maj(two[3], t4, t5);
                const uint32_t s1 = u0 ^ u1, f2 = u0 & u1;
                const uint32_t s2 = f0 ^ f1 ^ f2, s3 = maj(f0, f1, f2);
                tri = __popc(s0) + 2 * __popc(s1) + 4 * __popc(s2) + 8 * __popc(s3) - 2 * __popc(act);
                for (uint32_t m = s3 | (s2 & s1); m; m &= m - 1) tri -= 2 * s_extra[case_at(q, __ffs(m) - 1)];
            }
            // at most 32 x 32 x 12 of either in a segment
            uint32_t both = v | tri << 16;
            if (SHIFT == 5) {
                both = __reduce_add_sync(FULL, both);
            } else {
#pragma unroll
                for (uint32_t o = 1; o < per; o <<= 1) both += __shfl_xor_sync(FULL, both, o);
            }
            v = both & 0xFFFFu;
            tri = both >> 16;
        }
        if (writes) {
            A.segs[seg] = make_uint2(v, tri);
            if (tri) A.masks[seg] = SHIFT == 5 ? chunks : chunks >> first & ((1u << (per & 31u)) - 1u);
        }
        lo = hi;
        any_lo = any_hi;
        all_lo = all_hi;
    }
}

// ---------------------------------------------------------------- scanning ---
// Exclusive prefixes inside blocks of 4096 segments (vertices, triangles and
// active segments in one 64-bit scan), the blocks' totals, and the list of
// active segments: each block's part in order, the parts in any order, padded
// with empty entries to whole groups, so that a group's segments follow one
// another with nothing in between and their outputs are contiguous.
__global__ void __launch_bounds__(512) mc_cell_scan(CellArgs A) {
    __shared__ uint64_t s_w[16];
    __shared__ uint32_t s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();     // the counts
    pdl_trigger();
    const uint32_t i0 = blockIdx.x * SCAN_BLOCK_SEGS + threadIdx.x * 8;
    uint2 a[8];
    uint32_t mask[8] = {};  // (of a segment without triangles: anything)
    uint64_t sum = 0;  // vertices << 38 | triangles << 13 | active segments
    auto packed = [](uint2 c) { return ((uint64_t)c.x << 38) | ((uint64_t)c.y << 13) | (c.y ? 1u : 0u); };
    if (i0 + 8 <= A.nsegs) {
        const uint4* p = reinterpret_cast<const uint4*>(A.segs + i0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint4 q = p[k];
            a[2 * k] = make_uint2(q.x, q.y);
            a[2 * k + 1] = make_uint2(q.z, q.w);
        }
        const uint4* m = reinterpret_cast<const uint4*>(A.masks + i0);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint4 q = m[k];
            mask[4 * k] = q.x;
            mask[4 * k + 1] = q.y;
            mask[4 * k + 2] = q.z;
            mask[4 * k + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            a[k] = i0 + k < A.nsegs ? A.segs[i0 + k] : make_uint2(0, 0);
            if (a[k].y) mask[k] = A.masks[i0 + k];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) sum += packed(a[k]);
    uint64_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    uint64_t before = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < 16; ++w) {
        if (w < warp) before += s_w[w];
        all += s_w[w];
    }
    const uint32_t active = (uint32_t)all & 0x1FFFu, padded = (active + A.group - 1) / A.group * A.group;
    if (threadIdx.x == 0) {
        s_base = active ? atomicAdd(&A.ctrl[0], padded) : 0u;
        A.blocks[blockIdx.x] = make_uint2((uint32_t)(all >> 38), (uint32_t)(all >> 13) & 0x1FFFFFFu);
    }
    uint64_t run = before + incl - sum;
    __syncthreads();
    const uint32_t base = s_base;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint2 pre = make_uint2((uint32_t)(run >> 38), (uint32_t)(run >> 13) & 0x1FFFFFFu);
        if (i0 + k < A.nsegs) A.segs[i0 + k] = pre;
        if (a[k].y) A.list[base + ((uint32_t)run & 0x1FFFu)] = make_uint4(i0 + k, pre.x, pre.y, mask[k]);
        run += packed(a[k]);
    }
    if (active + threadIdx.x < padded) A.list[base + active + threadIdx.x] = make_uint4(0, 0, 0, 0);
}

// (vertices, triangles) of the scan blocks before `end`, in every lane
__device__ __forceinline__ uint2 blocks_before(const CellArgs& A, uint32_t end, uint32_t lane) {
    uint2 s = make_uint2(0, 0);
    for (uint32_t b = lane; b < end; b += 32) {
        const uint2 t = __ldcg(A.blocks + b);
        s.x += t.x;
        s.y += t.y;
    }
    return make_uint2(__reduce_add_sync(FULL, s.x), __reduce_add_sync(FULL, s.y));
}

// the grand totals, from one warp (overflow of 32 bits is an error)
__device__ __forceinline__ void write_totals(const CellArgs& A, uint32_t lane) {
    uint64_t v = 0, t = 0;
    for (uint32_t b = lane; b < A.nblocks; b += 32) {
        const uint2 c = __ldcg(A.blocks + b);
        v += c.x;
        t += c.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(FULL, v, o);
        t += __shfl_xor_sync(FULL, t, o);
    }
    if (lane == 0) {
        A.totals[0] = t;
        A.totals[1] = v;
        if (v > 0xFFFFFFFFull || t > 0xFFFFFFFFull) atomicOr(A.err, DERR_CAPACITY);
    }
}

// Mesh extents of every lattice of a table (first vertex, vertices, first
// triangle, triangles), a warp each, from the prefixes of its first segment
// and of the one after its last.
__global__ void __launch_bounds__(256) mc_cell_extents(CellArgs A, uint32_t ngrids, uint4* out) {
    const uint32_t lane = threadIdx.x & 31, i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= ngrids) return;
    auto prefix = [&](uint32_t seg) {
        const uint2 b = blocks_before(A, seg < A.nsegs ? seg / SCAN_BLOCK_SEGS : A.nblocks, lane);
        const uint2 p = seg < A.nsegs ? A.segs[seg] : make_uint2(0, 0);
        return make_uint2(b.x + p.x, b.y + p.y);
    };
    const uint2 a = prefix(A.grids[i].seg0), b = prefix(i + 1 < ngrids ? A.grids[i + 1].seg0 : A.nsegs);
    if (lane == 0) out[i] = make_uint4(a.x, b.x - a.x, a.y, b.y - a.y);
}

// ---------------------------------------------------------------- emission ---
struct CellEmitArgs {
    CellArgs c;
    float* out_v;
    uint32_t* out_i;
    uint64_t* out_k;
    uint64_t cap_v, cap_t;
    uint32_t* edge_id;  // vertex id per lattice edge, keyed by (upper end point * 3 + axis)
    // page-locked host buffers (device-side pointers, null: none) that also
    // receive the mesh when all of it fits both them and the device buffers
    float* host_v;
    uint64_t host_cap_v, host_cap_t;
};

// place of set bit number r (from 0, lowest first) of m
__device__ __forceinline__ uint32_t nth_bit(uint32_t m, uint32_t r) {
    uint32_t at = 0;
#pragma unroll
    for (uint32_t w = 16; w > 0; w >>= 1) {
        const uint32_t n = __popc(m & ((1u << w) - 1u));
        if (r >= n) {
            r -= n;
            m >>= w;
            at += w;
        }
    }
    return at;
}

// A warp's working set.
struct EmitStage {
    // 32 active chunks: the four sign rows' words with the next word's first
    // bit (padded, so that lanes reading different chunks hit different
    // banks), active cells, the exclusive prefix of their counts, the chunk's
    // row and place (y << 16 | c) and layer
    uint2 row[32][5];
    uint32_t act[32], excl[32], yc[32], z[32];
    // the lattice's cell edges: offsets of the two ends' values (in visiting
    // direction) and of the edge-map key, from corner 0's
    uint64_t uoff[12], voff[12];
    uint32_t koff[12];
    // a round of 32 cells: (lane << 4 | edge) of each new vertex and the lane of each triangle
    uint16_t vert[32 * 12];
    uint8_t tri[32 * 5 + 3];
};

// the ends of a cell edge in visiting direction, as offsets from corner 0
// (x | y << 1 | z << 2 of the first, << 3 of the second) and its axis << 6
__device__ __forceinline__ uint32_t edge_ends(uint32_t e) {
    const uint32_t u = __ldg(&iso_edge_connection[e][0]), v = __ldg(&iso_edge_connection[e][1]);
    return __ldg(&iso_corners[u][0]) | __ldg(&iso_corners[u][1]) << 1 | __ldg(&iso_corners[u][2]) << 2 |
           __ldg(&iso_corners[v][0]) << 3 | __ldg(&iso_corners[v][1]) << 4 | __ldg(&iso_corners[v][2]) << 5 |
           __ldg(&g_edge_axis[e]) << 6;
}

// A warp per group of listed segments: their active chunks are taken 32 at a
// time (lane = chunk), sign words and active cells staged in shared memory
// with their count prefix, and the chunks' active cells handed out 32 at a
// time in chunk order (lane = cell: its chunk by a binary search over the
// prefix).  The round's vertices, and then its triangles, are handed out one
// per lane in their turn (each cell notes its own in shared memory), so that
// lanes stay busy however many of either a cell has, and neighbouring lanes
// write neighbouring places.  Output offsets are the group's plus a running
// warp scan of the cells' counts (the reference's emission order).  Every
// vertex records its id in a dense per-lattice-edge map, and triangles are
// written as map keys; mc_resolve_ids then replaces each key by the id its
// owner recorded (the map needs no initialisation: every crossing edge has an
// owner, and only crossing edges are referenced).  Keys are 3 * (upper end
// point) + axis, so the (at most three) edges an interior cell owns, which
// all end at its corner 6, share one 12-byte slot.
template <bool TABLE>
__global__ void __launch_bounds__(256, 5) mc_cell_emit(CellEmitArgs A) {
    __shared__ EmitStage s_stage[8];
    // per sign pattern (two bits of each staged row): triangle edges, crossing
    // mask | triangle count << 12 | first-use ranks of edges 5, 6, 10 for
    // interior cells (iso_case_pack), case
    __shared__ uint4 s_case[256];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    EmitStage& S = s_stage[warp];
    {
        // rows (y, z) (y+1, z) (y, z+1) (y+1, z+1), bits x and x+1 -> CORNERS order
        const uint32_t r = threadIdx.x;
        const uint32_t cs = (r & 3) | ((r >> 3) & 1) << 2 | ((r >> 2) & 1) << 3 | ((r >> 4) & 3) << 4 |
                            ((r >> 7) & 1) << 6 | ((r >> 6) & 1) << 7;
        uint4 pk = __ldg(reinterpret_cast<const uint4*>(&iso_case_pack[cs]));
        pk.w = cs;
        s_case[r] = pk;
    }
    const uint32_t ends_l = edge_ends(min(lane, 11u));
    __syncthreads();
    pdl_wait();     // the list
    pdl_trigger();
    if (blockIdx.x == 0 && warp == 0) write_totals(A.c, lane);
    // a persistent grid: groups differ widely in cells, so each warp takes
    // another when it is done with one (blocks of a fixed group per warp left
    // warps idle behind their slowest: 41 against 62 % occupancy)
    const uint32_t ngroups = A.c.ctrl[0] / A.c.group;
    for (uint32_t grp = blockIdx.x * 8 + warp; grp < ngroups;) {
        uint32_t taken = 0;
        if (lane == 0) taken = atomicAdd(&A.c.ctrl[1], 1u);
        // lane e < group: entry e
        uint4 ent = make_uint4(0, 0, 0, 0);
        if (lane < A.c.group) ent = __ldcg(A.c.list + (size_t)grp * A.c.group + lane);
        const uint2 bp = blocks_before(A.c, __shfl_sync(FULL, ent.x, 0) / SCAN_BLOCK_SEGS, lane);
        uint32_t vcarry = bp.x + __shfl_sync(FULL, ent.y, 0), tcarry = bp.y + __shfl_sync(FULL, ent.z, 0);
        const uint32_t nch = __popc(ent.w), ech = warp_incl_scan(nch, lane) - nch;
        const uint32_t chunks = __reduce_add_sync(FULL, nch);
        for (uint32_t c0 = 0; c0 < chunks;) {
            // the entry of this lane's chunk: the last one that starts at or before it
            const uint32_t slot = c0 + lane;
            uint32_t e = 0;
            for (uint32_t k = 1; k < A.c.group; ++k)
                if (__shfl_sync(FULL, ech, k) <= slot) e = k;
            const uint32_t seg = __shfl_sync(FULL, ent.x, e), mask = __shfl_sync(FULL, ent.w, e);
            const uint32_t bit = nth_bit(mask, slot - __shfl_sync(FULL, ech, e));
            bool live = slot < chunks;
            uint32_t gi = 0, take = min(32u, chunks - c0);
            if (TABLE) {
                // the chunks of one lattice at a time
                gi = live ? __ldg(A.c.seg_grid + seg) : 0u;
                const uint32_t g0 = __shfl_sync(FULL, gi, 0);
                const uint32_t other = __ballot_sync(FULL, live && gi != g0);
                if (other) take = (uint32_t)__ffs(other) - 1;
                live = live && lane < take;
                gi = g0;
            }
            const Grid& g = TABLE ? A.c.grids[gi] : A.c.grid;
            uint32_t grid_v0 = 0;  // first vertex of this lattice's mesh
            if (TABLE) grid_v0 = __ldcg(&A.c.segs[g.seg0]).x + blocks_before(A.c, g.seg0 / SCAN_BLOCK_SEGS, lane).x;
            __syncwarp();  // the previous chunks are used
            uint32_t act = 0;
            {
                const uint32_t ls = seg - g.seg0, zc = fdiv(ls, g.div_sl);
                const uint32_t l = ((ls - zc * g.SL) << g.shift) + bit, y = fdiv(l, g.div_cw), c = l - y * g.CW;
                if (live) {
                    const uint32_t* a = g.bits + ((uint64_t)zc * g.ny + y) * g.W + c;
                    const uint32_t* b = a + (uint64_t)g.ny * g.W;
                    const bool nxt = c + 1 < g.W;
                    const uint32_t q0 = __ldg(a), n0 = nxt ? __ldg(a + 1) : 0u;
                    const uint32_t q1 = __ldg(a + g.W), n1 = nxt ? __ldg(a + g.W + 1) : 0u;
                    const uint32_t q2 = __ldg(b), n2 = nxt ? __ldg(b + 1) : 0u;
                    const uint32_t q3 = __ldg(b + g.W), n3 = nxt ? __ldg(b + g.W + 1) : 0u;
                    const uint32_t any = q0 | q1 | q2 | q3, all = q0 & q1 & q2 & q3;
                    const uint32_t any1 = __funnelshift_r(any, n0 | n1 | n2 | n3, 1);
                    const uint32_t all1 = __funnelshift_r(all, n0 & n1 & n2 & n3, 1);
                    act = (any | any1) & ~(all & all1) & chunk_valid(c, g.nx - 1);
                    S.row[lane][0] = make_uint2(q0, n0);
                    S.row[lane][1] = make_uint2(q1, n1);
                    S.row[lane][2] = make_uint2(q2, n2);
                    S.row[lane][3] = make_uint2(q3, n3);
                }
                S.yc[lane] = (y << 16) | c;
                S.z[lane] = zc;
                if (lane < 12 && (TABLE || c0 == 0)) {
                    auto at = [](uint32_t d, uint64_t row, uint64_t layer) {
                        return (d & 1) + ((d & 2) ? row : 0) + ((d & 4) ? layer : 0);
                    };
                    const uint32_t d = ends_l;
                    S.uoff[lane] = at(d, g.pitch, g.pitch * g.ny);
                    S.voff[lane] = at(d >> 3, g.pitch, g.pitch * g.ny);
                    S.koff[lane] = 3 * (uint32_t)at((d | d >> 3) & 7u, g.nx, (uint64_t)g.nx * g.ny) + (d >> 6);
                }
            }
            c0 += take;
            const uint32_t n = __popc(act), excl = warp_incl_scan(n, lane) - n;
            const uint32_t total = __reduce_add_sync(FULL, n);
            S.act[lane] = act;
            S.excl[lane] = excl;
            __syncwarp();
            for (uint32_t b0 = 0; b0 < total; b0 += 32) {
                const uint32_t kk = b0 + lane;
                uint32_t x = 0, yy = 0, z = 0, own = 0, nt = 0, te_lo = 0, te_hi = 0, rank = 0;
                bool inner = true;
                uint64_t rk = 0;
                if (kk < total) {
                    // the last chunk whose prefix is <= kk
                    uint32_t j = 0;
    #pragma unroll
                    for (uint32_t step = 16; step > 0; step >>= 1)
                        if (S.excl[j + step] <= kk) j += step;
                    const uint32_t i = nth_bit(S.act[j], kk - S.excl[j]);
                    uint32_t r = 0;
    #pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint2 q = S.row[j][k];
                        r |= (__funnelshift_r(q.x, q.y, i) & 3u) << (2 * k);
                    }
                    const uint32_t yc = S.yc[j];
                    yy = yc >> 16;
                    z = S.z[j];
                    x = 32 * (yc & 0xFFFFu) + i;
                    const uint4 pk = s_case[r];
                    te_lo = pk.x;
                    te_hi = pk.y;
                    nt = (pk.z >> 12) & 7u;
                    inner = x > 0 && yy > 0 && z > 0;
                    if (inner) {
                        own = pk.z & 0x460u;  // owned edges 5, 6, 10
                        rank = pk.z >> 16;
                    } else {
                        const int cls = (x == 0 ? 1 : 0) | (yy == 0 ? 2 : 0) | (z == 0 ? 4 : 0);
                        own = pk.z & __ldg(&iso_owned_mask[cls]);
                        rk = __ldg(&iso_owned_rank[cls][pk.w]);
                    }
                }
                // one scan for both counts: vertices (at most 12 x 32) | triangles << 16
                const uint32_t both = __popc(own) | nt << 16, bi = warp_incl_scan(both, lane), be = bi - both;
                const uint32_t round = __shfl_sync(FULL, bi, 31), vn = round & 0xFFFFu, tn = round >> 16;
                const uint32_t vpre = be & 0xFFFFu, tpre = be >> 16;
                // owned edges, by their rank in the cell's order of first use
                if (inner) {
                    if (own & 0x020u) S.vert[vpre + (rank & 15u)] = (uint16_t)(lane << 4 | 5);
                    if (own & 0x040u) S.vert[vpre + (rank >> 4 & 15u)] = (uint16_t)(lane << 4 | 6);
                    if (own & 0x400u) S.vert[vpre + (rank >> 8 & 15u)] = (uint16_t)(lane << 4 | 10);
                } else {
                    for (uint32_t m = own; m; m &= m - 1) {
                        const uint32_t k = __ffs(m) - 1;
                        S.vert[vpre + ((uint32_t)(rk >> (4 * k)) & 15u)] = (uint16_t)(lane << 4 | k);
                    }
                }
    #pragma unroll
                for (uint32_t k = 0; k < 5; ++k)
                    if (k < nt) S.tri[tpre + k] = (uint8_t)lane;
                __syncwarp();
                const uint32_t yx = (yy << 16) | x;
                for (uint32_t v0 = 0; v0 < vn; v0 += 32) {
                    const uint32_t j = v0 + lane, code = S.vert[min(j, vn - 1)], src = code >> 4, k = code & 15u;
                    const uint32_t cyx = __shfl_sync(FULL, yx, src), cz = __shfl_sync(FULL, z, src);
                    const uint32_t d = __shfl_sync(FULL, ends_l, k);
                    if (j >= vn) continue;
                    const uint32_t cx = cyx & 0xFFFFu, cy = cyx >> 16;
                    // Signed::find_crossing_point (distance.rs:64-69) on the
                    // edge, in the visiting cell's direction
                    const float* val = g.values + (((uint64_t)cz * g.ny + cy) * g.pitch + cx);
                    const float fa = __ldg(val + S.uoff[k]), fb = __ldg(val + S.voff[k]);
                    const uint32_t cell = (cz * g.ny + cy) * g.nx + cx;
                    V3 pa, pb;
                    if (g.positions) {
                        const float4* pos = g.positions + cell;
                        const uint32_t lay = g.nx * g.ny;
                        const float4 qa = __ldg(pos + ((d & 1) + ((d & 2) ? g.nx : 0) + ((d & 4) ? lay : 0)));
                        const float4 qb = __ldg(pos + ((d >> 3 & 1) + ((d & 16) ? g.nx : 0) + ((d & 32) ? lay : 0)));
                        pa = v3(qa.x, qa.y, qa.z);
                        pb = v3(qb.x, qb.y, qb.z);
                    } else {
                        const uint32_t gz = cz + g.zoff;
                        pa = v3((float)(cx + (d & 1)) * g.inv, (float)(cy + (d >> 1 & 1)) * g.inv,
                                (float)(gz + (d >> 2 & 1)) * g.inv);
                        pb = v3((float)(cx + (d >> 3 & 1)) * g.inv, (float)(cy + (d >> 4 & 1)) * g.inv,
                                (float)(gz + (d >> 5 & 1)) * g.inv);
                    }
                    const float delta = fb - fa;
                    const float tt = (delta == 0.0f) ? 0.5f : -fa / delta;
                    const float omt = 1.0f - tt;
                    const uint32_t vid = vcarry + j;
                    if (vid < A.cap_v) {
                        float* o = A.out_v + 3 * (size_t)vid;
                        o[0] = pa.x * omt + pb.x * tt;
                        o[1] = pa.y * omt + pb.y * tt;
                        o[2] = pa.z * omt + pb.z * tt;
                        if (A.out_k) {
                            // the lattice edge's key: lower end point * 3 + axis
                            const uint32_t lo = d & d >> 3 & 7u;
                            A.out_k[2 * (size_t)vid] =
                                (((uint64_t)(cz + (lo >> 2) + g.zoff) * g.ny + cy + (lo >> 1 & 1)) * g.nx + cx + (lo & 1)) * 3 +
                                (d >> 6);
                            A.out_k[2 * (size_t)vid + 1] = 0;
                        }
                    } else {
                        atomicOr(A.c.err, DERR_CAPACITY);
                    }
                    A.edge_id[g.edge0 + 3 * cell + S.koff[k]] = vid - grid_v0;
                }
                // triangles (march_cube, marching_cubes_impl.rs:102-117) as edge-map
                // keys, resolved to vertex ids once every owner has written its ids
                const uint32_t key0 = g.edge0 + 3 * ((z * g.ny + yy) * g.nx + x);
                for (uint32_t t0 = 0; t0 < tn; t0 += 32) {
                    const uint32_t j = t0 + lane, src = S.tri[min(j, tn - 1)];
                    const uint32_t k = j - __shfl_sync(FULL, tpre, src), key = __shfl_sync(FULL, key0, src);
                    const uint64_t te = (uint64_t)__shfl_sync(FULL, te_hi, src) << 32 | __shfl_sync(FULL, te_lo, src);
                    if (j >= tn) continue;
                    const uint32_t w = (uint32_t)(te >> (12 * k)), t = tcarry + j;
                    if (t < A.cap_t) {
                        uint32_t* o = A.out_i + 3 * (size_t)t;
                        o[0] = key + S.koff[w & 15u];
                        o[1] = key + S.koff[w >> 4 & 15u];
                        o[2] = key + S.koff[w >> 8 & 15u];
                    } else {
                        atomicOr(A.c.err, DERR_CAPACITY);
                    }
                }
                vcarry += vn;
                tcarry += tn;
                __syncwarp();  // the round's notes are used
            }
        }
        if (A.host_v) {
            // the group's vertices, just written by this warp, in whole lines to
            // the host (the warp's own stores are ordered before its reads)
            const uint2 all = blocks_before(A.c, A.c.nblocks, lane);
            if (all.x <= A.host_cap_v && all.y <= A.host_cap_t && all.x <= A.cap_v && all.y <= A.cap_t) {
                __syncwarp();
                const uint32_t vbase = bp.x + __shfl_sync(FULL, ent.y, 0);
                const size_t f0 = 3 * (size_t)vbase, f1 = 3 * (size_t)vcarry;
                for (size_t f = f0 + lane; f < f1; f += 32) A.host_v[f] = __ldcg(A.out_v + f);
            }
        }
        grp = gridDim.x * 8 + __shfl_sync(FULL, taken, 0);
    }
}
