// ExtendedMarchingCubes::new(size).extract (src/extended_marching_cubes.rs:
// 51-93) on the device.  The work of each lattice point and cell is in
// emc.cuh; here each pass is one grid-stride launch over its items, the
// counts are scanned over blocks of cells (block_sums.cuh), and the host reads
// the two totals once to size the mesh.
//
//   emc_sample     Directed value of every lattice point (float4 per point)
//                  and one sign bit per point
//   emc_active     case of every cell, from the sign bits; the cells with
//                  corners on both sides go to a list, which the later passes
//                  walk instead of the grid
//   emc_count      feature decision per active cell; vertices and triangles
//                  of every block of 1024 cells; the feature cells go to a
//                  second list with their tangent planes
//   emc_features   the feature points (MinimiseQEF), a few cells per warp, on
//                  a side stream beside everything below but the last pass
//   scan_block_sums  first vertex and first triangle of every block
//   emc_offsets    those of every active cell
//   emc_vertices   owned edge vertices; the edge map
//   emc_triangles  marching-cubes triangles and fans, in traversal order
//   emc_flips      feature-edge rotations
//   emc_points     the feature points to their places among the vertices
#include <cuda_runtime.h>

#include <algorithm>

#include "block_sums.cuh"
#include "internal.h"
#include "qef_rows.cuh"

#define ISO_TABLE static __device__ const
#include "emc_tables.h"
#include "mc_tables.h"

// The host halves of emc.cuh's functions are compiled here too, reading this
// unit's device tables; only the host build of the same functions (for the
// tests, with host tables) calls them.
#pragma nv_diag_suppress 20091
#include "emc.cuh"
#pragma nv_diag_default 20091

namespace iso {
namespace {

constexpr uint32_t BLOCK_CELLS = 1024;  // cells with one entry in the scan
// feature cells whose tangent planes and points are kept, per lattice line:
// sharp edges are curves, so their cells grow with the size, not its square (a
// box with a sphere and a torus at 128: 2200 cells, 17 per line; at 48 the room
// is 11 KB per line).  Cells beyond it are solved after the scan, by
// emc_points.
constexpr uint32_t FEATURES_PER_LINE = 48;

// emc_count's result for a feature cell, and emc_features'
struct Feature {
    emc::PlanesN planes;
    qef::F3 point;
};

// device counters of one extraction
struct Ctrl {
    uint32_t active, features;
    uint2 totals;  // vertices, triangles
    unsigned long long flips;
};

// Sign bit i & 31 of word i >> 5: lattice point i is inside.  A lane takes
// four points, 32 apart (128 solid: 62 us a point at a time).
constexpr uint32_t POINTS = 4;
__global__ void __launch_bounds__(256) emc_sample(emc::Args A, uint32_t points, uint32_t* bits) {
    constexpr uint32_t span = 256 * POINTS;
    for (uint32_t i0 = blockIdx.x * span; i0 < points; i0 += gridDim.x * span) {
        const uint32_t i = i0 + (threadIdx.x >> 5) * 32 * POINTS + (threadIdx.x & 31);
        V3 q[POINTS], v[POINTS];
#pragma unroll
        for (uint32_t j = 0; j < POINTS; ++j) q[j] = emc::item_pos(A.g, i + 32 * j);
        emc::eval_vectors<POINTS>(A.prog, q, v);
#pragma unroll
        for (uint32_t j = 0; j < POINTS; ++j) {
            const uint32_t at = i + 32 * j;
            const bool in = at < points;
            if (in) A.field[at] = make_float4(v[j].x, v[j].y, v[j].z, 0.0f);
            const uint32_t word = __ballot_sync(0xFFFFFFFFu, in && emc::directed_inside(v[j]));
            if ((threadIdx.x & 31) == 0 && in) bits[at >> 5] = word;
        }
    }
}

// Every cell's case, from two neighbouring sign bits in each of its four rows
// (reading the eight values themselves was 16 times the bytes); the cells
// with corners on both sides (the only ones with work in the later passes)
// are appended to `list` in any order.
__global__ void __launch_bounds__(256) emc_active(emc::Args A, uint32_t cells, const uint32_t* bits, uint32_t* list,
                                                  Ctrl* ctrl) {
    const uint32_t lane = threadIdx.x & 31, n = A.g.n;
    for (uint32_t c0 = blockIdx.x * 256; c0 < cells; c0 += gridDim.x * 256) {
        const uint32_t c = c0 + threadIdx.x;
        bool active = false;
        if (c < cells) {
            uint32_t x, y, z;
            emc::cell_xyz(n, c, &x, &y, &z);
            // points i and i + 1; the word after the last one is allocated
            auto pair = [&](uint32_t i) {
                const uint32_t* w = bits + (i >> 5);
                return __funnelshift_r(__ldg(w), __ldg(w + 1), i & 31) & 3u;
            };
            const uint32_t p = (z * n + y) * n + x;
            const uint32_t a = pair(p), b = pair(p + n), d = pair(p + n * n), e = pair(p + n * n + n);
            // corners 0-1-2-3 go round a face (marching_cubes_tables.rs:16-25)
            const uint32_t cube = a | (b & 2u) << 1 | (b & 1u) << 3 | d << 4 | (e & 2u) << 5 | (e & 1u) << 7;
            active = cube != 0 && cube != 255;
            A.cell[c] = (uint16_t)cube;
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, active);
        if (m) {
            const uint32_t leader = (uint32_t)__ffs(m) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&ctrl->active, (uint32_t)__popc(m));
            base = __shfl_sync(0xFFFFFFFFu, base, leader);
            if (active) list[base + __popc(m & ((1u << lane) - 1u))] = c;
        }
    }
}

// The feature decision of every active cell, four lanes to a cell: the
// program's normal at a crossing is the long chain here, a cell has three to
// twelve of them and there are too few active cells to hide it, so each lane
// takes every fourth crossing (one thread per cell, with its crossings in
// local memory, took 58 us for a solid at 128).
__global__ void __launch_bounds__(128) emc_count(emc::Args A, const uint32_t* list, Ctrl* ctrl, uint32_t* features,
                                                 Feature* kept, uint32_t cap, unsigned long long* sums) {
    __shared__ qef::F3 vtx[32][12], nrm[32][12];
    const uint32_t n = ctrl->active, sub = threadIdx.x & 3, g = threadIdx.x >> 2;
    for (uint32_t i0 = blockIdx.x * 32; i0 < n; i0 += gridDim.x * 32) {
        const uint32_t i = i0 + g;
        const bool live = i < n;
        uint32_t c = 0, x = 0, y = 0, z = 0;
        int cube = 0, count = 0;
        if (live) {
            c = list[i];
            cube = A.cell[c];
            emc::cell_xyz(A.g.n, c, &x, &y, &z);
            const uint32_t mask = iso_edge_mask[cube];
            count = __popc(mask);
            uint32_t rest = mask;
            for (int k = 0; k < count; ++k, rest &= rest - 1) {
                if ((k & 3) != (int)sub) continue;
                const V3 p = emc::edge_crossing(A, x, y, z, __ffs(rest) - 1);
                V3 nn;
                eval_hermite(A.prog, p, &nn);
                vtx[g][k] = qef::f3(p.x, p.y, p.z);
                nrm[g][k] = qef::normalised_or_zero(qef::f3(nn.x, nn.y, nn.z));
            }
        }
        __syncwarp();
        // TangentPlanes (tangent_planes_n): the pair of normals with the
        // smallest product, the first in (i, j) order of equals, each lane
        // over a quarter of the rows i
        float least = emc::F32_MAX;
        uint32_t pair = ~0u;
        for (int r = (int)sub; r < count; r += 4)
            for (int k = 0; k < count; ++k) {
                const float angle = qef::dot(nrm[g][r], nrm[g][k]);
                if (angle < least) {
                    least = angle;
                    pair = (uint32_t)(16 * r + k);
                }
            }
        for (uint32_t o = 1; o < 4; o <<= 1) {
            const float a2 = __shfl_xor_sync(0xFFFFFFFFu, least, o);
            const uint32_t p2 = __shfl_xor_sync(0xFFFFFFFFu, pair, o);
            if (a2 < least || (a2 == least && p2 < pair)) {
                least = a2;
                pair = p2;
            }
        }
        if (live && sub == 0) {
            const uint32_t feature = !(least > qef::FEATURE_ANGLE);
            uint32_t nv, nt;
            emc::cell_counts(x, y, z, cube, feature, &nv, &nt);
            atomicAdd(sums + c / BLOCK_CELLS, (unsigned long long)nt << 32 | nv);
            if (feature) {
                A.cell[c] = (uint16_t)(cube | 256);
                const uint32_t at = atomicAdd(&ctrl->features, 1u);
                features[at] = c;
                if (at < cap) {
                    const qef::F3 axis = pair == ~0u ? qef::f3(0.0f, 0.0f, 0.0f)
                                                     : qef::cross(nrm[g][pair >> 4], nrm[g][pair & 15]);
                    emc::planes_about(vtx[g], nrm[g], count, least, axis, &kept[at].planes);
                }
            }
        }
        __syncwarp();
    }
}

// First vertex and first triangle of every active cell (nothing reads those
// of the others): a thread block per block of cells, four cells per thread.
__global__ void __launch_bounds__(256) emc_offsets(emc::Args A, uint32_t cells, const unsigned long long* sums) {
    const unsigned long long base = sums[blockIdx.x];
    if (base == NO_ITEMS) return;
    const uint32_t c0 = blockIdx.x * BLOCK_CELLS + 4 * threadIdx.x;
    unsigned long long v[4], mine = 0;
    for (uint32_t k = 0; k < 4; ++k) {
        v[k] = 0;
        if (c0 + k >= cells) continue;
        const uint32_t info = A.cell[c0 + k];
        const int cube = (int)(info & 255);
        if (cube == 0 || cube == 255) continue;
        uint32_t x, y, z, nv, nt;
        emc::cell_xyz(A.g.n, c0 + k, &x, &y, &z);
        emc::cell_counts(x, y, z, cube, info >> 8, &nv, &nt);
        v[k] = (unsigned long long)nt << 32 | nv;
        mine += v[k];
    }
    unsigned long long run = offset_in_block(base, mine);
    for (uint32_t k = 0; k < 4; ++k) {
        if (v[k]) {
            A.voff[c0 + k] = (uint32_t)run;
            A.toff[c0 + k] = (uint32_t)(run >> 32);
        }
        run += v[k];
    }
}

// every vertex but the feature points
__global__ void __launch_bounds__(128) emc_vertices(emc::Args A, const uint32_t* list, const Ctrl* ctrl) {
    const uint32_t n = ctrl->active;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        emc::vertex_item(A, list[i], false);
}

// The feature points of the kept feature cells, over one-warp blocks, as soon
// as the cells are known.  Each is one serial chain of f64 operations (the
// SVD, in the reference's order), and a warp's f64 instruction holds its
// sub-partition's f64 unit for many cycles whatever its active lanes.  Few
// cells go to eight lanes each (qef_rows.cuh; a cell with more than eight
// crossings to its first lane), which shortens the chain; more, beyond a warp
// of four cells for each sub-partition, to one lane each, in full warps (dc.cu
// has a case measured there).  128 solid, 2200 cells: 72 us, 92 with a lane
// each, spread evenly.
constexpr uint32_t ROW_WARPS = 4;  // one-warp blocks per SM
__global__ void __launch_bounds__(32) emc_features(emc::Args A, Feature* kept, uint32_t cap, const Ctrl* ctrl) {
    const uint32_t n = min(ctrl->features, cap);
    if (n <= 4 * gridDim.x) {
        const uint32_t group = threadIdx.x >> 3, y = threadIdx.x & 7, i = 4 * blockIdx.x + group;
        if (i >= n) return;
        const emc::PlanesN& t = kept[i].planes;
        const int rows = t.n;
        bool ok = true;
        if (rows <= 8) {
            const uint32_t at = min(y, (uint32_t)rows - 1);
            const qef::F3 p = qef::add(t.com, qef::solve_planes_rows(0xFFu << (8 * group), t.normal[at], t.d[at], rows,
                                                                     t.feature == qef::EDGE, &ok));
            if (y == 0) kept[i].point = p;
        } else if (y == 0) {
            kept[i].point = emc::minimise_qef_n(t, &ok);
        }
        if (!ok && y == 0) atomicOr(A.err, DERR_SVD_ITER);
        return;
    }
    for (uint32_t i = blockIdx.x * 32 + threadIdx.x; i < n; i += gridDim.x * 32) {
        bool ok;
        const qef::F3 p = emc::minimise_qef_n(kept[i].planes, &ok);
        if (!ok) atomicOr(A.err, DERR_SVD_ITER);
        kept[i].point = p;
    }
}

// the feature points to the first vertex of their cells; those of the cells
// that were not kept are found here
__global__ void __launch_bounds__(32) emc_points(emc::Args A, const uint32_t* features, const Feature* kept, uint32_t cap,
                                                 uint32_t n) {
    for (uint32_t i = blockIdx.x * 32 + threadIdx.x; i < n; i += gridDim.x * 32) {
        const uint32_t c = features[i];
        if (i < cap) emc::put_vertex(A, A.voff[c], kept[i].point);
        else emc::feature_item(A, c);
    }
}

__global__ void __launch_bounds__(256) emc_triangles(emc::Args A, const uint32_t* list, const Ctrl* ctrl) {
    const uint32_t n = ctrl->active;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        emc::triangle_item(A, list[i]);
}

// a flip's first face is a feature cell's
__global__ void __launch_bounds__(64) emc_flips(emc::Args A, const uint32_t* features, uint32_t n, Ctrl* ctrl) {
    uint32_t mine = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        mine += emc::flip_item(A, features[i]);
    mine = __reduce_add_sync(0xFFFFFFFFu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&ctrl->flips, (unsigned long long)mine);
}

enum : uint32_t {
    OP_PT_DOMAIN_H = 0x01, OP_PT_TRANSLATE_H = 0x02, OP_PT_POP_H = 0x04,
    OP_SPHERE_H = 0x10, OP_BOX_H = 0x11, OP_CYLINDER_H = 0x12, OP_TORUS_H = 0x13,
    OP_UNION_H = 0x20, OP_INTERSECTION_H = 0x21, OP_DIFFERENCE_H = 0x22, OP_CD_BEGIN_H = 0x40, OP_CD_END_H = 0x41,
};

// The reference defines sample_vector (the Directed metric) for its
// primitives, Union, Intersection, Difference and CentralDifference; the
// translate and domain-map point ops move the point as they do for values.
bool directed_ops_only(const iso_program* p) {
    for (uint32_t w : p->ops) {
        switch (w & 0xFF) {
        case OP_PT_DOMAIN_H: case OP_PT_TRANSLATE_H: case OP_PT_POP_H:
        case OP_SPHERE_H: case OP_BOX_H: case OP_CYLINDER_H: case OP_TORUS_H:
        case OP_UNION_H: case OP_INTERSECTION_H: case OP_DIFFERENCE_H:
        case OP_CD_BEGIN_H: case OP_CD_END_H:
            break;
        default:
            return false;
        }
    }
    return true;
}

unsigned grid_for(const iso_ctx* ctx, uint64_t items, unsigned threads, unsigned per_sm) {
    const uint64_t want = (items + threads - 1) / threads;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)ctx->sms * per_sm));
}

}  // namespace
}  // namespace iso

using namespace iso;

// everything after the scan; leaves the counters in h_pinned[0 .. 2] and the
// error flags in h_pinned[3]
static iso_status emc_emit(iso_ctx* ctx, emc::Args A, uint64_t cells, uint32_t nblocks, uint32_t cap,
                           const uint32_t* active, const uint32_t* features, const Feature* kept, Ctrl* ctrl,
                           const unsigned long long* sums) {
    iso_status s;
    cudaError_t e = cudaMemcpyAsync(ctx->h_pinned, ctrl, 16, cudaMemcpyDeviceToHost, ctx->stream);
    {
        StageTimer timer(ctx, ISO_STAGE_CLASSIFY);
        emc_offsets<<<nblocks, 256, 0, ctx->stream>>>(A, (uint32_t)cells, sums);
        ctx->launches++;
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "emc counts");
    const Ctrl* h = (const Ctrl*)ctx->h_pinned;
    const uint32_t nactive = h->active, nfeat = h->features;
    if ((s = ensure(ctx, ctx->mesh_v, 12ull * h->totals.x + 16)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->mesh_i, 12ull * h->totals.y + 16)) != ISO_OK) return s;
    A.vertices = (float*)ctx->mesh_v.p;
    A.indices = (uint32_t*)ctx->mesh_i.p;
    A.cap_v = h->totals.x;
    A.cap_t = h->totals.y;
    if (nactive) {
        StageTimer timer(ctx, ISO_STAGE_EMIT);  // (without the wait for the side stream)
        emc_vertices<<<grid_for(ctx, nactive, 128, 32), 128, 0, ctx->stream>>>(A, active, ctrl);
        emc_triangles<<<grid_for(ctx, nactive, 256, 16), 256, 0, ctx->stream>>>(A, active, ctrl);
        ctx->launches += 2;
        if (nfeat) {
            emc_flips<<<grid_for(ctx, nfeat, 64, 32), 64, 0, ctx->stream>>>(A, features, nfeat, ctrl);
            ctx->launches++;
        }
    }
    if (nfeat) {
        if ((s = join_side(ctx)) != ISO_OK) return s;
        StageTimer timer(ctx, ISO_STAGE_EMIT);
        emc_points<<<grid_for(ctx, nfeat, 32, 32), 32, 0, ctx->stream>>>(A, features, kept, cap, nfeat);
        ctx->launches++;
    }
    if ((s = check_launch(ctx, "emc emit")) != ISO_OK) return s;
    e = cudaMemcpyAsync(ctx->h_pinned + 2, &ctrl->flips, 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_pinned + 3, ctx->d_err, 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? ISO_OK : cuda_fail(ctx, e, "emc emit");
}

static iso_status emc_extract_impl(iso_ctx* ctx, const iso_program* prog, uint32_t size, iso_mesh_info* info,
                                   uint64_t* flips_out) {
    if (prog->ctx != ctx) return fail(ctx, ISO_ERR_INVALID_ARG, "program belongs to another context");
    if (size > 513) return fail(ctx, ISO_ERR_TOO_LARGE, "ExtendedMarchingCubes size above 513");
    if (!directed_ops_only(prog))
        return fail(ctx, ISO_ERR_INVALID_ARG,
                    "ExtendedMarchingCubes needs the Directed metric: primitives, Union, Intersection, Difference, "
                    "translate, domain map and CentralDifference only");
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    ctx->last = iso_mesh_info{};
    ctx->last_flags = 0;
    ctx->last_vertex_floats = 3;
    if (size < 2) {  // no cell
        if (info) *info = ctx->last;
        return ISO_OK;
    }
    const uint32_t n = size;
    const uint64_t points = emc::num_points(n), cells = emc::num_cells(n);
    const uint32_t nblocks = (uint32_t)((cells + BLOCK_CELLS - 1) / BLOCK_CELLS);
    const uint32_t cap = (uint32_t)std::min<uint64_t>(cells, (uint64_t)FEATURES_PER_LINE * n);
    const uint64_t bit_words = (((points + 31) / 32 + 1) + 63) & ~(uint64_t)63;
    // Directed field | case + feature per cell | counters and the blocks'
    // sums, vertex and triangle offsets | edge map
    if ((s = ensure(ctx, ctx->field, 16 * points)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->aux, 2 * cells)) != ISO_OK) return s;
    const size_t ctrl_bytes = sizeof(Ctrl) + 8ull * nblocks;
    if ((s = ensure(ctx, ctx->scan, ctrl_bytes + 8 * cells)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->edges, 12 * points)) != ISO_OK) return s;
    // the active cells, the feature cells, sign bits, the kept features
    const uint64_t list_words = (cells + 63) & ~(uint64_t)63;
    if ((s = ensure(ctx, ctx->aux2, 4 * (2 * list_words + bit_words) + sizeof(Feature) * (uint64_t)cap)) != ISO_OK) return s;
    uint32_t* active = (uint32_t*)ctx->aux2.p;
    uint32_t* features = active + list_words;
    uint32_t* bits = features + list_words;
    Feature* kept = (Feature*)(bits + bit_words);
    Ctrl* ctrl = (Ctrl*)ctx->scan.p;
    unsigned long long* sums = (unsigned long long*)(ctrl + 1);

    emc::Args A{};
    A.prog = prog->view();
    A.g = emc::Grid{n, 1.0f / (float)(n - 1)};
    A.field = (float4*)ctx->field.p;
    A.cell = (uint16_t*)ctx->aux.p;
    A.voff = (uint32_t*)(sums + nblocks);
    A.toff = A.voff + cells;
    A.edge_map = (uint32_t*)ctx->edges.p;
    A.err = ctx->d_err;
    cudaError_t e = cudaMemsetAsync(ctrl, 0, ctrl_bytes, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "emc counters");
    {
        StageTimer timer(ctx, ISO_STAGE_SAMPLE);
        emc_sample<<<grid_for(ctx, points, 256 * POINTS, 16), 256, 0, ctx->stream>>>(A, (uint32_t)points, bits);
    }
    cudaStream_t side;
    {
        StageTimer timer(ctx, ISO_STAGE_CLASSIFY);
        emc_active<<<grid_for(ctx, cells, 256, 16), 256, 0, ctx->stream>>>(A, (uint32_t)cells, bits, active, ctrl);
        emc_count<<<grid_for(ctx, cells, 32, 16), 128, 0, ctx->stream>>>(A, active, ctrl, features, kept, cap, sums);
        ctx->launches += 3;
        if ((s = check_launch(ctx, "emc count")) != ISO_OK) return s;
        // the feature points on a side stream: the passes below neither read
        // nor wait for them
        if ((s = fork_side(ctx, &side)) != ISO_OK) return s;
        {
            StageTimer features_timer(ctx, ISO_STAGE_EMIT, side);
            emc_features<<<ROW_WARPS * (unsigned)std::max(ctx->sms, 1), 32, 0, side>>>(A, kept, cap, ctrl);
        }
        scan_block_sums<<<1, 1024, 0, ctx->stream>>>(sums, nblocks, &ctrl->totals);
        ctx->launches += 2;
    }
    s = emc_emit(ctx, A, cells, nblocks, cap, active, features, kept, ctrl, sums);
    if (ctx->side_open) {  // the passes ended early
        const iso_status j = join_side(ctx);
        if (s == ISO_OK) s = j;
    }
    if (s != ISO_OK) return s;
    const uint64_t nv = ctx->h_pinned[1] & 0xFFFFFFFFu, nt = ctx->h_pinned[1] >> 32, nflips = ctx->h_pinned[2];
    if ((uint32_t)ctx->h_pinned[3] && (s = read_device_errors(ctx)) != ISO_OK) return s;
    ctx->last.num_vertices = nv;
    ctx->last.num_triangles = nt;
    ctx->last.num_cells = cells;
    if (flips_out) *flips_out = nflips;
    if (info) *info = ctx->last;
    return ISO_OK;
}

// ISO_FLAG_NORMALS: IndexedInterleavedNormals, sample_normal at every vertex
extern "C" iso_status iso_emc_extract(iso_ctx* ctx, const iso_program* prog, uint32_t size, uint32_t flags,
                                      iso_mesh_info* info, uint64_t* flips) {
    iso::NvtxRange nvtx_range("iso_emc_extract");
    if (!ctx || !prog) return ISO_ERR_INVALID_ARG;
    if (flags & ~(uint32_t)ISO_FLAG_NORMALS) return fail(ctx, ISO_ERR_INVALID_ARG, "unsupported flags");
    iso_status s = emc_extract_impl(ctx, prog, size, info, flips);
    if (s != ISO_OK || !(flags & ISO_FLAG_NORMALS)) return s;
    if ((s = attach_normals(ctx, prog)) != ISO_OK) return s;
    if (info) *info = ctx->last;
    return ISO_OK;
}
