// Batched MarchingCubes: thousands of independent chunks, each a
// MarchingCubes::new(size_i).extract over its own source, in one pass.
//
// * Sampling: the culled sampler of bricks.cuh (sign bits everywhere, values
//   where marching cubes can read them, primitives pruned per sub-brick) in
//   two launches: a warp classifies up to 32 sub-bricks of one chunk and
//   lists the mixed ones, and a persistent grid evaluates the list, four
//   sub-bricks of one chunk to a warp.  Warps do not cross a chunk's z-slabs;
//   the slab depth per chunk-size class is the whole chunk unless
//   iso_batch_set_slab or iso_batch_autotune chooses another.
// * Counting, scan and emission: the cell passes of mc_cells.cuh over a table
//   of grids that share one edge map; when the grids' edges do not fit its
//   32-bit keys, or there is no memory for it (4 B per lattice edge), the
//   block emit over grids whose 32-cell chunks are laid out range-aligned in
//   one global index space (mc_chunk.cuh).
// * iso_batch_run with ISO_BATCH_GRAPH captures all of it in one CUDA graph
//   and replays it; output capacities come from the previous run (the first
//   run is eager and sizes them), and an overflow is detected on the device
//   and answered with an eager re-run.
// * iso_batch_run_per_chunk runs the same chunks one extraction at a time
//   (sample, count, scan, emit, with the host syncs of iso_mc_extract) and
//   concatenates the meshes: the comparison point for the batch.
//
// Output: the context's mesh holds all chunks' vertices and triangles
// back to back; indices are local to each chunk (each chunk is its own
// IndexedVertices mesh); iso_batch_extents gives each chunk's
// (first vertex, vertices, first triangle, triangles).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "bricks.cuh"
#include "internal.h"
#include "vm.cuh"

namespace iso {
// defined in mc.cu
iso_status mc_extract_grids(iso_ctx* ctx, const void* d_grids, uint32_t ngrids, const uint32_t* d_range_grid,
                            uint32_t chunks, uint32_t max_cw, void* scratch, uint64_t cap_v, uint64_t cap_t,
                            float* out_v, uint32_t* out_i, uint32_t* extents, uint64_t* totals, bool sync_sizes);
size_t mc_grid_bytes();
void mc_fill_grid(void* dst, const Lattice& L, uint32_t chunk0, uint32_t* nchunks, uint32_t* cw);
size_t mc_grids_scratch_bytes(uint32_t chunks, uint32_t ngrids);
struct CellTable;
CellTable* mc_table_create(iso_ctx* ctx, const Lattice* L, uint32_t n);
void mc_table_destroy(CellTable* t);
uint64_t mc_table_edges(const CellTable* t);
iso_status mc_extract_table(iso_ctx* ctx, const CellTable* t, uint64_t cap_v, uint64_t cap_t, float* out_v,
                            uint32_t* out_i, uint32_t* extents, uint64_t* totals, bool sync_sizes);
}  // namespace iso

using namespace iso;

namespace {

struct SampleGrid {
    ProgView pv;
    uint32_t n;  // MarchingCubes::new(n): n x n x (n+1) samples
    float inv;
    float* field;
    uint64_t pitch;
    uint32_t* bits;
    uint32_t W;
};

// Up to eight groups of four sub-bricks along x (32 x 4 x 4 samples) of one
// grid, from group `first` in (z, y, x) order: a classifying warp's work.
struct Task {
    uint32_t grid, first, groups;
};

// A mixed sub-brick: its grid, its place sx | sy << 8 | sz << 17 (NO_BRICK:
// none, filling up a warp's four) and the primitives it keeps.
struct Mixed {
    uint32_t grid, at;
    uint64_t keep;
};
constexpr uint32_t NO_BRICK = 0xFFFFFFFFu;
constexpr uint32_t HELD = 16;  // primitives whose values a classifying lane keeps in shared memory

__device__ __forceinline__ BrickLattice lattice_of(const SampleGrid& sg) {
    return BrickLattice{sg.pv.lip, sg.pv.slack, sg.n,     sg.n,  sg.n + 1, sg.inv,
                        sg.field,  sg.pitch,    sg.bits, sg.W, 0,        1.0f};
}

// A warp per task, a lane per sub-brick: no barrier, and no lane waits for
// another grid's primitives.  (Blocks that classified a tile, listed its
// mixed sub-bricks in shared memory and sampled them between barriers spent
// 44 % of their warps' time at those, on tiles of 20 sub-bricks for a 16^3
// chunk: 495 us for 1024 chunks of 16^3 to 64^3 cells; now 39 and 139 for
// batch_rows, which issues in 73 % of its slots.)
__global__ void __launch_bounds__(256) batch_classify(const Task* tasks, const SampleGrid* grids, uint32_t ntasks,
                                                      uint32_t ngrids, Mixed* list, uint32_t* count, uint32_t* err) {
    __shared__ float s_held[HELD][256];
    const uint32_t lane = threadIdx.x & 31, t = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (t >= ntasks) return;
    const Task k = tasks[t];
    if (k.grid >= ngrids) {  // warp-uniform
        if (lane == 0) atomicOr(err, DERR_TABLE);
        return;
    }
    const SampleGrid sg = grids[k.grid];
    const BrickLattice g = lattice_of(sg);
    const VmEval ev{sg.pv};
    const uint32_t SY = (g.ny + 3) / 4, gi = k.first + (lane >> 2), j = lane & 3;
    const bool have = (lane >> 2) < k.groups;
    const uint32_t w = gi % g.W, sy = gi / g.W % SY, sz = gi / (g.W * SY), sx = 4 * w + j;
    const uint32_t xa = 8 * sx, ya = 4 * sy, za = 4 * sz;
    uint32_t cls = BRICK_MIXED;
    uint64_t keep = ~0ull;
    if (!have || (g.lip > 0.0f && xa >= g.nx)) cls = BRICK_OUT;  // no samples: sign bits stay clear
    else if (g.lip > 0.0f)
        cls = brick_class(ev, g, xa, min(xa + 7, g.nx - 1), ya, min(ya + 3, g.ny - 1), za, min(za + 3, g.nz - 1), &keep,
                          &s_held[0][threadIdx.x], HELD, 256);
    const uint32_t mixed = __ballot_sync(0xFFFFFFFFu, cls == BRICK_MIXED);
    // the group's sign words: its four lanes take four rows each
    uint32_t cls4 = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) cls4 |= __shfl_sync(0xFFFFFFFFu, cls, (lane & ~3u) + i) << (8 * i);
    if (have) {
        // (the mixed sub-bricks' bytes are batch_rows' to write, after this)
        const uint32_t word = decided_word(cls4, g.nx, w), z = za + j;
        for (uint32_t y = ya; y < min(ya + 4, g.ny) && z < g.nz; ++y) g.bits[((uint64_t)z * g.ny + y) * g.W + w] = word;
    }
    if (!mixed) return;
    // the task's part of the list, filled up to whole fours
    const uint32_t n = __popc(mixed), padded = (n + 3) & ~3u;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(count, padded);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (cls == BRICK_MIXED)
        list[base + __popc(mixed & ((1u << lane) - 1u))] = Mixed{k.grid, sx | sy << 8 | sz << 17, keep};
    if (lane < padded - n) list[base + n + lane] = Mixed{k.grid, NO_BRICK, 0};
}

// The listed sub-bricks, four of one grid to a warp, over a persistent grid.
__global__ void __launch_bounds__(256) batch_rows(const SampleGrid* grids, const Mixed* list, const uint32_t* count) {
    const uint32_t n = *count, lane = threadIdx.x & 31;
    for (uint32_t q = 4 * (blockIdx.x * 8 + (threadIdx.x >> 5)); q < n; q += 32 * gridDim.x) {
        const Mixed m = list[q + (lane >> 3)];
        const SampleGrid& sg = grids[__shfl_sync(0xFFFFFFFFu, m.grid, 0)];
        const BrickLattice g = lattice_of(sg);
        const bool have = m.at != NO_BRICK;
        const uint32_t sx = have ? m.at & 255u : 0u, ya = have ? 4 * (m.at >> 8 & 511u) : 0u,
                       za = have ? 4 * (m.at >> 17) : 0u;
        brick_fill(VmEval{sg.pv}, g, have, sx, ya, za, g.ny, g.nz, warp_or64(m.keep));
    }
}

// The tasks of one chunk of `n` (n x n x (n + 1) samples) for slab depth
// `depth` (0: the whole chunk), rounded up to whole sub-bricks (4 layers).
template <class F>
void chunk_tasks(uint32_t grid, uint32_t n, uint32_t depth, F&& add) {
    const uint32_t layer = words_per_row(n) * ((n + 3) / 4), nsz = (n + 1 + 3) / 4;  // groups per four layers
    const uint32_t zg = depth ? std::min((depth + 3) / 4, nsz) : nsz;
    for (uint32_t z = 0; z < nsz; z += zg) {
        const uint32_t end = layer * std::min(z + zg, nsz);
        for (uint32_t first = layer * z; first < end; first += 8) add(Task{grid, first, std::min(8u, end - first)});
    }
}

struct Chunk {
    uint32_t prog, size;
};

}  // namespace

struct iso_batch {
    iso_ctx* ctx = nullptr;
    std::vector<const iso_program*> programs;
    std::vector<Chunk> chunks;
    std::vector<uint32_t> slab;      // slab depth per chunk (0 = whole grid)
    // device layout
    void* arena = nullptr;
    size_t arena_bytes = 0;
    SampleGrid* d_sgrids = nullptr;
    void* d_grids = nullptr;
    uint32_t* d_range_grid = nullptr;
    Task* d_tasks = nullptr;  // the sampler's tasks, then room for their mixed sub-bricks
    uint32_t ntasks = 0;
    uint32_t* d_next = nullptr;  // how many mixed sub-bricks are listed
    uint32_t* d_extents = nullptr;   // 4 per chunk
    uint64_t* d_totals = nullptr;    // [0] triangles [1] vertices
    void* d_scratch = nullptr;       // chunk-pass scratch
    uint32_t total_chunks = 0, max_cw = 0;
    std::vector<SampleGrid> sgrids;
    std::vector<uint32_t> grid_chunk0;
    // outputs and graph
    uint64_t cap_v = 0, cap_t = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // the context's mesh buffers the graph was captured with: another
    // extraction on the context may regrow (free and reallocate) them
    void* graph_v = nullptr;
    void* graph_i = nullptr;
    void* graph_e = nullptr;  // its edge map (null: captured with the block emit)
    CellTable* table = nullptr;
    bool sized = false;
    // iso_batch_run_per_chunk_async: each chunk as a grid of its own
    void* d_solo_grids = nullptr;
    std::vector<uint32_t> solo_chunks, solo_cw;
};

namespace {

// where the list of mixed sub-bricks starts behind `n` tasks
size_t list_at(size_t n) { return (sizeof(Task) * n + 255) & ~(size_t)255; }

// Device copy of `tasks`, with room for every sub-brick of theirs behind it.
cudaError_t upload_tasks(iso_ctx* ctx, const std::vector<Task>& tasks, Task** d_tasks) {
    const size_t n = tasks.size();
    cudaError_t e = cudaMalloc((void**)d_tasks, list_at(n) + 32 * sizeof(Mixed) * std::max<size_t>(n, 1));
    if (e == cudaSuccess && n) e = upload(ctx, *d_tasks, tasks.data(), sizeof(Task) * n);
    return e;
}

iso_status build_tasks(iso_batch* b) {
    std::vector<Task> tasks;
    for (uint32_t i = 0; i < b->chunks.size(); ++i)
        chunk_tasks(i, b->chunks[i].size, b->slab[i], [&](const Task& t) { tasks.push_back(t); });
    if (b->d_tasks) cudaFree(b->d_tasks);
    b->d_tasks = nullptr;
    b->ntasks = (uint32_t)tasks.size();
    cudaError_t e = upload_tasks(b->ctx, tasks, &b->d_tasks);
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    return e == cudaSuccess ? ISO_OK : cuda_fail(b->ctx, e, "tasks");
}

// the culled sampler over `ntasks` tasks
cudaError_t launch_sampler(const iso_batch* b, const Task* d_tasks, uint32_t ntasks) {
    const cudaStream_t stream = b->ctx->stream;
    cudaError_t e = cudaMemsetAsync(b->d_next, 0, 4, stream);
    if (e != cudaSuccess) return e;
    Mixed* list = (Mixed*)((char*)d_tasks + list_at(ntasks));
    batch_classify<<<(ntasks + 7) / 8, 256, 0, stream>>>(d_tasks, b->d_sgrids, ntasks, (uint32_t)b->chunks.size(), list,
                                                         b->d_next, b->ctx->d_err);
    batch_rows<<<persistent_blocks(b->ctx, (const void*)batch_rows), 256, 0, stream>>>(b->d_sgrids, list, b->d_next);
    return cudaGetLastError();
}

// the sampler's best time of three over `tasks`, after a first run
cudaError_t time_sampler(const iso_batch* b, const std::vector<Task>& tasks, cudaEvent_t begin, cudaEvent_t end,
                         float* best) {
    Task* d_tasks = nullptr;
    cudaError_t e = upload_tasks(b->ctx, tasks, &d_tasks);
    *best = 1e30f;
    for (int rep = 0; rep < 4 && e == cudaSuccess; ++rep) {
        float ms = 0.0f;
        e = cudaEventRecord(begin, b->ctx->stream);
        if (e == cudaSuccess) e = launch_sampler(b, d_tasks, (uint32_t)tasks.size());
        if (e == cudaSuccess) e = cudaEventRecord(end, b->ctx->stream);
        if (e == cudaSuccess) e = cudaEventSynchronize(end);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, begin, end);
        if (rep > 0) *best = std::min(*best, ms);
    }
    if (d_tasks) cudaFree(d_tasks);
    return e;
}

struct EventPair {
    cudaEvent_t begin = nullptr, end = nullptr;
    ~EventPair() {
        if (begin) cudaEventDestroy(begin);
        if (end) cudaEventDestroy(end);
    }
};

// whether the cell passes can run: the table exists and the edge map is there
bool edge_map_ready(iso_batch* b) {
    if (!b->table) return false;
    if (ensure(b->ctx, b->ctx->edges, 4 * mc_table_edges(b->table)) == ISO_OK) return true;
    cudaGetLastError();
    b->ctx->last_error.clear();
    return false;
}

// enqueue the whole batch on the context's stream (sync_sizes: the counts are
// read back before the emit)
iso_status enqueue(iso_batch* b, bool cells, bool sync_sizes) {
    iso_ctx* ctx = b->ctx;
    {
        StageTimer timer(ctx, ISO_STAGE_SAMPLE);
        cudaError_t e = launch_sampler(b, b->d_tasks, b->ntasks);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "batch sampler");
    }
    ctx->launches += 2;
    if (cells)
        return mc_extract_table(ctx, b->table, b->cap_v, b->cap_t, (float*)ctx->mesh_v.p, (uint32_t*)ctx->mesh_i.p,
                                b->d_extents, b->d_totals, sync_sizes);
    return mc_extract_grids(ctx, b->d_grids, (uint32_t)b->chunks.size(), b->d_range_grid, b->total_chunks, b->max_cw,
                            b->d_scratch, b->cap_v, b->cap_t, (float*)ctx->mesh_v.p, (uint32_t*)ctx->mesh_i.p,
                            b->d_extents, b->d_totals, sync_sizes);
}

// stored: the totals and the error flags are in h_pinned already (the cell passes)
iso_status finish(iso_batch* b, bool stored, iso_mesh_info* info) {
    iso_ctx* ctx = b->ctx;
    cudaError_t e = cudaSuccess;
    if (!stored) {
        e = cudaMemcpyAsync(ctx->h_pinned, b->d_totals, 16, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_pinned + 2, ctx->d_err, 4, cudaMemcpyDeviceToHost, ctx->stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "batch totals");
    const uint64_t nt = ctx->h_pinned[0], nv = ctx->h_pinned[1];
    uint64_t cells = 0;
    for (auto& c : b->chunks) cells += (uint64_t)(c.size - 1) * (c.size - 1) * c.size;
    ctx->last.num_vertices = nv;
    ctx->last.num_triangles = nt;
    ctx->last.num_cells = cells;
    ctx->last_flags = 0;
    ctx->last_vertex_floats = 3;
    if (info) *info = ctx->last;
    if ((uint32_t)ctx->h_pinned[2]) return read_device_errors(ctx);
    return ISO_OK;
}

}  // namespace

extern "C" {

iso_status iso_batch_create(iso_ctx* ctx, const iso_program* const* programs, uint32_t nprograms,
                            const iso_chunk_desc* chunks, uint32_t nchunks, iso_batch** out) {
    if (!ctx || !out || (!programs && nprograms) || (!chunks && nchunks) || nchunks == 0) return ISO_ERR_INVALID_ARG;
    *out = nullptr;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    iso_batch* b = new iso_batch();
    b->ctx = ctx;
    b->programs.assign(programs, programs + nprograms);
    for (uint32_t i = 0; i < nprograms; ++i)
        if (!programs[i] || programs[i]->ctx != ctx) {
            delete b;
            return fail(ctx, ISO_ERR_INVALID_ARG, "null program or program of another context");
        }
    for (uint32_t i = 0; i < nchunks; ++i) {
        if (chunks[i].program >= nprograms || chunks[i].size < 2 || chunks[i].size > 1025) {
            delete b;
            return fail(ctx, ISO_ERR_INVALID_ARG, "chunk program index out of range or size not in [2, 1025]");
        }
        b->chunks.push_back(Chunk{chunks[i].program, chunks[i].size});
    }
    b->slab.assign(nchunks, 0);
    // layout: per chunk field + bits; grid tables; chunk-pass scratch
    size_t off = 0;
    auto take = [&](size_t bytes) {
        off = (off + 255) & ~(size_t)255;
        const size_t at = off;
        off += bytes;
        return at;
    };
    std::vector<size_t> field_off(nchunks), bits_off(nchunks);
    uint32_t chunk0 = 0;
    b->grid_chunk0.resize(nchunks);
    for (uint32_t i = 0; i < nchunks; ++i) {
        const uint32_t n = b->chunks[i].size;
        field_off[i] = take(4ull * default_pitch(n) * n * (n + 1));
        bits_off[i] = take(4ull * words_per_row(n) * n * (n + 1));
        const uint32_t cw = (n - 1 + 31) / 32;
        const uint32_t nch = cw * (n - 1) * n;
        b->grid_chunk0[i] = chunk0;
        chunk0 += (nch + 255) / 256 * 256;
        b->max_cw = std::max(b->max_cw, cw);
    }
    b->total_chunks = chunk0;
    const uint32_t nranges = chunk0 / 256;
    const size_t sg_off = take(sizeof(SampleGrid) * nchunks);
    const size_t g_off = take(mc_grid_bytes() * nchunks);
    const size_t rg_off = take(4ull * nranges);
    const size_t next_off = take(256);
    const size_t ext_off = take(16ull * nchunks);
    const size_t tot_off = take(64);
    const size_t scr_off = take(mc_grids_scratch_bytes(b->total_chunks, nchunks));
    b->arena_bytes = off;
    cudaError_t e = cudaMalloc(&b->arena, b->arena_bytes);
    if (e != cudaSuccess) {
        delete b;
        return cuda_fail(ctx, e, "batch arena");
    }
    char* base = (char*)b->arena;
    b->d_sgrids = (SampleGrid*)(base + sg_off);
    b->d_grids = base + g_off;
    b->d_range_grid = (uint32_t*)(base + rg_off);
    b->d_next = (uint32_t*)(base + next_off);
    b->d_extents = (uint32_t*)(base + ext_off);
    b->d_totals = (uint64_t*)(base + tot_off);
    b->d_scratch = base + scr_off;
    std::vector<char> grids(mc_grid_bytes() * nchunks);
    std::vector<uint32_t> range_grid(nranges);
    std::vector<Lattice> lattices;
    b->sgrids.resize(nchunks);
    for (uint32_t i = 0; i < nchunks; ++i) {
        const uint32_t n = b->chunks[i].size;
        const iso_program* p = b->programs[b->chunks[i].prog];
        SampleGrid sg{p->view(), n, 1.0f / (float)(n - 1), (float*)(base + field_off[i]), default_pitch(n),
                      (uint32_t*)(base + bits_off[i]), words_per_row(n)};
        b->sgrids[i] = sg;
        Lattice L{n, n, n + 1, default_pitch(n), sg.field, sg.bits, sg.W, sg.inv, nullptr};
        lattices.push_back(L);
        uint32_t nch = 0, cw = 0;
        mc_fill_grid(grids.data() + mc_grid_bytes() * i, L, b->grid_chunk0[i], &nch, &cw);
        for (uint32_t r = b->grid_chunk0[i] / 256; r < (b->grid_chunk0[i] + nch + 255) / 256; ++r) range_grid[r] = i;
    }
    e = upload(ctx, b->d_sgrids, b->sgrids.data(), sizeof(SampleGrid) * nchunks);
    if (e == cudaSuccess) e = upload(ctx, b->d_grids, grids.data(), grids.size());
    if (e == cudaSuccess && nranges) e = upload(ctx, b->d_range_grid, range_grid.data(), 4ull * nranges);
    if (e != cudaSuccess) {
        iso_batch_destroy(b);
        return cuda_fail(ctx, e, "batch tables");
    }
    if ((s = build_tasks(b)) != ISO_OK) {
        iso_batch_destroy(b);
        return s;
    }
    b->table = mc_table_create(ctx, lattices.data(), nchunks);
    *out = b;
    return ISO_OK;
}

iso_status iso_batch_destroy(iso_batch* b) {
    if (!b) return ISO_ERR_INVALID_ARG;
    cudaSetDevice(b->ctx->device);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->d_tasks) cudaFree(b->d_tasks);
    mc_table_destroy(b->table);
    if (b->arena) cudaFree(b->arena);
    if (b->d_solo_grids) cudaFree(b->d_solo_grids);
    delete b;
    return ISO_OK;
}

iso_status iso_batch_set_slab(iso_batch* b, uint32_t size, uint32_t depth) {
    if (!b) return ISO_ERR_INVALID_ARG;
    for (size_t i = 0; i < b->chunks.size(); ++i)
        if (size == 0 || b->chunks[i].size == size) b->slab[i] = depth;
    return build_tasks(b);
}

iso_status iso_batch_run(iso_batch* b, uint32_t flags, iso_mesh_info* info) {
    iso::NvtxRange nvtx_range("iso_batch_run");
    if (!b) return ISO_ERR_INVALID_ARG;
    iso_ctx* ctx = b->ctx;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    const bool graph = (flags & ISO_BATCH_GRAPH) != 0;
    const bool cells = edge_map_ready(b);
    if (!graph || !b->sized) {
        // eager: sizes are read back between the count and the emit passes
        s = enqueue(b, cells, true);
        if (s != ISO_OK) return s;
        if ((s = finish(b, cells, info)) != ISO_OK) return s;
        if (!b->sized || ctx->last.num_vertices > b->cap_v || ctx->last.num_triangles > b->cap_t) {
            b->cap_v = ctx->last.num_vertices + ctx->last.num_vertices / 4 + 1024;
            b->cap_t = ctx->last.num_triangles + ctx->last.num_triangles / 4 + 1024;
            b->sized = true;
            if (b->exec) {
                cudaGraphExecDestroy(b->exec);
                b->exec = nullptr;
            }
            if (b->graph) {
                cudaGraphDestroy(b->graph);
                b->graph = nullptr;
            }
        }
        return ISO_OK;
    }
    if ((s = ensure(ctx, ctx->mesh_v, 12 * b->cap_v)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->mesh_i, 12 * b->cap_t)) != ISO_OK) return s;
    void* const edges = cells ? ctx->edges.p : nullptr;
    if (b->exec && (b->graph_v != ctx->mesh_v.p || b->graph_i != ctx->mesh_i.p || b->graph_e != edges)) {
        cudaGraphExecDestroy(b->exec);
        cudaGraphDestroy(b->graph);
        b->exec = nullptr;
        b->graph = nullptr;
    }
    if (!b->exec) {
        cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "begin capture");
        const bool timing = ctx->timing;
        ctx->timing = false;  // no events inside the graph
        s = enqueue(b, cells, false);
        ctx->timing = timing;
        cudaGraph_t g = nullptr;
        e = cudaStreamEndCapture(ctx->stream, &g);
        if (s != ISO_OK) {
            if (g) cudaGraphDestroy(g);
            return s;
        }
        if (e != cudaSuccess) return cuda_fail(ctx, e, "end capture");
        b->graph = g;
        e = cudaGraphInstantiate(&b->exec, g, 0);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "instantiate graph");
        b->graph_v = ctx->mesh_v.p;
        b->graph_i = ctx->mesh_i.p;
        b->graph_e = edges;
    }
    {
        StageTimer timer(ctx, ISO_STAGE_OTHER);
        cudaError_t e = cudaGraphLaunch(b->exec, ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "graph launch");
    }
    ctx->launches += 7;
    s = finish(b, cells, info);
    if (s == ISO_ERR_CAPACITY || ctx->last.num_vertices > b->cap_v || ctx->last.num_triangles > b->cap_t) {
        b->sized = false;  // grow and run eagerly
        return iso_batch_run(b, 0, info);
    }
    return s;
}

iso_status iso_batch_run_per_chunk(iso_batch* b, iso_mesh_info* info) {
    iso::NvtxRange nvtx_range("iso_batch_run_per_chunk");
    if (!b) return ISO_ERR_INVALID_ARG;
    iso_ctx* ctx = b->ctx;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    // each chunk through the single-grid path, then appended to the batch output
    std::vector<uint32_t> ext(4 * b->chunks.size());
    uint64_t nv = 0, nt = 0;
    std::vector<float> hv;
    std::vector<uint32_t> hi;
    if ((s = ensure(ctx, ctx->aux3, 12 * std::max<uint64_t>(b->cap_v, 1 << 20) + 12 * std::max<uint64_t>(b->cap_t, 1 << 20))) != ISO_OK)
        return s;
    uint64_t cap_v = ctx->aux3.bytes / 24, cap_t = ctx->aux3.bytes / 24;
    float* out_v = (float*)ctx->aux3.p;
    uint32_t* out_i = (uint32_t*)((char*)ctx->aux3.p + 12 * cap_v);
    for (size_t i = 0; i < b->chunks.size(); ++i) {
        const SampleGrid& g = b->sgrids[i];
        const uint32_t n = g.n;
        if ((s = launch_sample_grid(ctx, b->programs[b->chunks[i].prog], n, n, n + 1, g.inv, g.field, g.pitch,
                                    g.bits, true)) != ISO_OK)
            return s;
        Lattice L{n, n, n + 1, g.pitch, g.field, g.bits, g.W, g.inv, nullptr};
        iso_mesh_info mi;
        if ((s = mc_extract_lattice(ctx, L, 0, &mi)) != ISO_OK) return s;
        if (nv + mi.num_vertices > cap_v || nt + mi.num_triangles > cap_t)
            return fail(ctx, ISO_ERR_CAPACITY, "per-chunk output arena too small");
        cudaMemcpyAsync(out_v + 3 * nv, ctx->mesh_v.p, 12 * mi.num_vertices, cudaMemcpyDeviceToDevice, ctx->stream);
        cudaMemcpyAsync(out_i + 3 * nt, ctx->mesh_i.p, 12 * mi.num_triangles, cudaMemcpyDeviceToDevice, ctx->stream);
        ext[4 * i + 0] = (uint32_t)nv;
        ext[4 * i + 1] = (uint32_t)mi.num_vertices;
        ext[4 * i + 2] = (uint32_t)nt;
        ext[4 * i + 3] = (uint32_t)mi.num_triangles;
        nv += mi.num_vertices;
        nt += mi.num_triangles;
    }
    // hand the concatenated mesh over as the context's mesh
    if ((s = ensure(ctx, ctx->mesh_v, 12 * std::max<uint64_t>(nv, 1))) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->mesh_i, 12 * std::max<uint64_t>(nt, 1))) != ISO_OK) return s;
    cudaMemcpyAsync(ctx->mesh_v.p, out_v, 12 * nv, cudaMemcpyDeviceToDevice, ctx->stream);
    cudaMemcpyAsync(ctx->mesh_i.p, out_i, 12 * nt, cudaMemcpyDeviceToDevice, ctx->stream);
    cudaMemcpyAsync(b->d_extents, ext.data(), 4 * ext.size(), cudaMemcpyHostToDevice, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "per-chunk run");
    uint64_t cells = 0;
    for (auto& c : b->chunks) cells += (uint64_t)(c.size - 1) * (c.size - 1) * c.size;
    ctx->last = iso_mesh_info{nv, nt, cells};
    ctx->last_flags = 0;
    ctx->last_vertex_floats = 3;
    if (info) *info = ctx->last;
    return ISO_OK;
}

iso_status iso_batch_run_per_chunk_async(iso_batch* b, iso_mesh_info* info) {
    iso::NvtxRange nvtx_range("iso_batch_run_per_chunk_async");
    if (!b) return ISO_ERR_INVALID_ARG;
    iso_ctx* ctx = b->ctx;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    if (!b->sized) return fail(ctx, ISO_ERR_INVALID_ARG, "run the batch once first (it sizes every chunk's output)");
    const uint32_t n_ch = (uint32_t)b->chunks.size();
    if (!b->d_solo_grids) {
        // every chunk as a grid of its own, chunk ids from 0
        std::vector<char> grids(mc_grid_bytes() * n_ch);
        b->solo_chunks.resize(n_ch);
        b->solo_cw.resize(n_ch);
        for (uint32_t i = 0; i < n_ch; ++i) {
            const SampleGrid& g = b->sgrids[i];
            Lattice L{g.n, g.n, g.n + 1, g.pitch, g.field, g.bits, g.W, g.inv, nullptr};
            mc_fill_grid(grids.data() + mc_grid_bytes() * i, L, 0, &b->solo_chunks[i], &b->solo_cw[i]);
        }
        cudaError_t e = cudaMalloc(&b->d_solo_grids, grids.size());
        if (e == cudaSuccess) e = upload(ctx, b->d_solo_grids, grids.data(), grids.size());
        if (e != cudaSuccess) return cuda_fail(ctx, e, "per-chunk grids");
    }
    // each chunk's output place and size, from the last run of the batch
    std::vector<uint32_t> ext(4ull * n_ch);
    cudaError_t e = cudaMemcpyAsync(ext.data(), b->d_extents, 16ull * n_ch, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "chunk extents");
    const uint64_t nv = (uint64_t)ext[4ull * (n_ch - 1)] + ext[4ull * (n_ch - 1) + 1];
    const uint64_t nt = (uint64_t)ext[4ull * (n_ch - 1) + 2] + ext[4ull * (n_ch - 1) + 3];
    if ((s = ensure(ctx, ctx->mesh_v, 12 * std::max<uint64_t>(nv, 1))) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->mesh_i, 12 * std::max<uint64_t>(nt, 1))) != ISO_OK) return s;
    float* out_v = (float*)ctx->mesh_v.p;
    uint32_t* out_i = (uint32_t*)ctx->mesh_i.p;
    uint32_t* dummy_extents = (uint32_t*)(b->d_totals + 4);  // [0, 16) of the totals block's unused half
    uint64_t* totals = b->d_totals;
    // per chunk: its sampler, count, scan and emit, queued back to back
    for (uint32_t i = 0; i < n_ch; ++i) {
        const SampleGrid& g = b->sgrids[i];
        if ((s = launch_sample_grid(ctx, b->programs[b->chunks[i].prog], g.n, g.n, g.n + 1, g.inv, g.field, g.pitch,
                                    g.bits, true)) != ISO_OK)
            return s;
        if ((s = mc_extract_grids(ctx, (const char*)b->d_solo_grids + mc_grid_bytes() * i, 1, nullptr,
                                  b->solo_chunks[i], b->solo_cw[i], b->d_scratch, ext[4ull * i + 1],
                                  ext[4ull * i + 3], out_v + 3ull * ext[4ull * i], out_i + 3ull * ext[4ull * i + 2],
                                  dummy_extents, totals, false)) != ISO_OK)
            return s;
    }
    e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "per-chunk run");
    if ((s = read_device_errors(ctx)) != ISO_OK) return s;
    uint64_t cells = 0;
    for (auto& c : b->chunks) cells += (uint64_t)(c.size - 1) * (c.size - 1) * c.size;
    ctx->last = iso_mesh_info{nv, nt, cells};
    ctx->last_flags = 0;
    ctx->last_vertex_floats = 3;
    if (info) *info = ctx->last;
    return ISO_OK;
}

iso_status iso_batch_extents(iso_batch* b, uint32_t* extents) {
    if (!b || !extents) return ISO_ERR_INVALID_ARG;
    iso_ctx* ctx = b->ctx;
    cudaError_t e = cudaMemcpyAsync(extents, b->d_extents, 16ull * b->chunks.size(), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? ISO_OK : cuda_fail(ctx, e, "extents");
}

iso_status iso_batch_autotune(iso_batch* b, const char* cache_path, uint32_t* chosen) {
    if (!b) return ISO_ERR_INVALID_ARG;
    iso_ctx* ctx = b->ctx;
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, ctx->device);
    // cached depths are for this sampler design on this GPU model
    const std::string gpu = std::string(prop.name) + " brick list";
    std::map<uint32_t, uint32_t> classes;  // size -> chunk count
    for (auto& c : b->chunks) classes[c.size]++;
    std::map<uint32_t, uint32_t> best;
    // cache lines: "<gpu>|<size>|<depth>"
    if (cache_path) {
        if (FILE* f = std::fopen(cache_path, "r")) {
            char line[512];
            while (std::fgets(line, sizeof(line), f)) {
                // (a line without both numbers is passed over)
                unsigned size = 0, depth = 0;
                if (std::strncmp(line, gpu.c_str(), gpu.size()) == 0 &&
                    std::sscanf(line + gpu.size(), "|%u|%u", &size, &depth) == 2)
                    best[size] = depth;
            }
            std::fclose(f);
        }
    }
    const uint32_t candidates[] = {4, 8, 16, 0};
    EventPair events;
    cudaError_t e = cudaEventCreate(&events.begin);
    if (e == cudaSuccess) e = cudaEventCreate(&events.end);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "autotune events");
    bool wrote = false;
    for (auto& cl : classes) {
        if (best.count(cl.first)) continue;
        float best_ms = 1e30f;
        uint32_t best_depth = 0;
        for (uint32_t d : candidates) {
            // time the sampler on this class's chunks only, slab depth d
            std::vector<Task> tasks;
            for (uint32_t i = 0; i < b->chunks.size(); ++i) {
                if (b->chunks[i].size != cl.first) continue;
                chunk_tasks(i, cl.first, d, [&](const Task& t) { tasks.push_back(t); });
            }
            float ms;
            e = time_sampler(b, tasks, events.begin, events.end, &ms);
            if (e != cudaSuccess) {
                cudaGetLastError();
                return cuda_fail(ctx, e, "autotune");
            }
            if (ms < best_ms) {
                best_ms = ms;
                best_depth = d;
            }
        }
        best[cl.first] = best_depth;
        wrote = true;
    }
    if (wrote && (s = read_device_errors(ctx)) != ISO_OK) return s;
    if (cache_path && wrote) {
        if (FILE* f = std::fopen(cache_path, "a")) {
            for (auto& kv : best) std::fprintf(f, "%s|%u|%u\n", gpu.c_str(), kv.first, kv.second);
            std::fclose(f);
        }
    }
    for (size_t i = 0; i < b->chunks.size(); ++i) b->slab[i] = best[b->chunks[i].size];
    if (chosen) {
        size_t k = 0;
        for (auto& kv : best) {
            chosen[2 * k] = kv.first;
            chosen[2 * k + 1] = kv.second;
            ++k;
        }
    }
    return build_tasks(b);
}

}  // extern "C"
