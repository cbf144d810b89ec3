// Culled sampling in the library: the device code of bricks_core.cuh with
// the library's program evaluator (vm.cuh), and the launch helpers.  The
// same core also runs with a per-program compiled evaluator (jit.cu).
#pragma once
#include <cuda_runtime.h>


#include "internal.h"
#include "vm.cuh"
#include "bricks_core.cuh"

namespace iso {

static_assert(BRICK_ERR_CAPACITY == DERR_CAPACITY, "the core's capacity bit is the library's");

// A set bit of a mask of primitives.  The union over a subset (in the same
// order) equals eval_prims wherever every dropped primitive's value exceeds
// some kept one's: fminf returns one of its operands, so the minimum over a
// subset that holds the minimiser is the minimum over all.
__device__ __forceinline__ uint32_t lowest_bit(uint64_t m) { return (uint32_t)(__ffsll((long long)m) - 1); }

// eval_scalar at N points
template <int N>
__device__ __forceinline__ void eval_scalars(const ProgView& pv, const V3 (&p)[N], float (&v)[N]) {
    V3 q[N];
    if (!pv.prims) {
#pragma unroll
        for (int j = 0; j < N; ++j) q[j] = p[j];
        eval_points<N>(pv, 0, pv.n_ops, q, v);
        return;
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        q[j] = prims_point(pv, p[j]);
        v[j] = pv.nprims ? __int_as_float(0x7FFFFFFF) : 0.0f;  // fminf takes the first primitive's value
    }
    for (uint32_t i = 0; i < pv.nprims; ++i) {
        const float4 c = ld_ro(pv.prims + 2 * i), a = ld_ro(pv.prims + 2 * i + 1);
        auto each = [&](auto&& sd) {
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = fminf(v[j], sd(v3(q[j].x - c.x, q[j].y - c.y, q[j].z - c.z)));
        };
        const uint32_t type = float_bits(c.w);
        if (type == OP_SPHERE) each([&](V3 t) { return sd_sphere(t, a.x); });
        else if (type == OP_BOX) each([&](V3 t) { return sd_box(t, a.x, a.y, a.z); });
        else if (type == OP_CYLINDER) each([&](V3 t) { return sd_cylinder(t, a.x, a.y); });
        else each([&](V3 t) { return sd_torus(t, a.x, a.y); });
    }
}

// The interpreted evaluator: the program's ops, or its flat list of
// translated primitives (pruned per sub-brick when there are at most 64).
struct VmEval {
    ProgView pv;
    __device__ __forceinline__ float value(V3 p) const { return eval_scalar(pv, p); }
    __device__ __forceinline__ bool prunable() const { return pv.prims != nullptr && pv.nprims <= BRICK_PRUNE_MAX; }
    __device__ __forceinline__ uint32_t nprims() const { return pv.nprims; }
    __device__ __forceinline__ V3 point(V3 p) const { return prims_point(pv, p); }
    __device__ __forceinline__ float prim(uint32_t i, V3 q) const { return prim_at(pv, i, q); }
    __device__ __forceinline__ void values_kept(uint64_t keep, const V3 (&p)[4], float (&v)[16]) const {
        V3 q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = point(p[j]);
        // fminf returns its other operand for a NaN, so the first primitive's value replaces it
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = __int_as_float(0x7FFFFFFF);
        for (; keep; keep &= keep - 1) {
            const uint32_t i = lowest_bit(keep);
            const float4 c = ld_ro(pv.prims + 2 * i), a = ld_ro(pv.prims + 2 * i + 1);
            auto each = [&](auto&& sd) {
#pragma unroll
                for (int r = 0; r < 16; ++r)
                    v[r] = fminf(v[r], sd(v3(q[0].x - c.x, q[r & 3].y - c.y, q[r >> 2].z - c.z)));
            };
            const uint32_t type = float_bits(c.w);
            if (type == OP_SPHERE) each([&](V3 t) { return sd_sphere(t, a.x); });
            else if (type == OP_BOX) each([&](V3 t) { return sd_box(t, a.x, a.y, a.z); });
            else if (type == OP_CYLINDER) each([&](V3 t) { return sd_cylinder(t, a.x, a.y); });
            else each([&](V3 t) { return sd_torus(t, a.x, a.y); });
        }
    }
};

// The culling bounds of a program for a lattice.
inline BrickLattice brick_lattice(const iso_program* prog, uint32_t nx, uint32_t ny, uint32_t nz, float inv,
                                  float* field, uint64_t pitch, uint32_t* bits, uint32_t W, uint32_t zoff,
                                  float reach_steps) {
    return BrickLattice{prog->lip, prog->slack, nx, ny, nz, inv, field, pitch, bits, W, zoff, reach_steps};
}

template <class Tiles>
__global__ void __launch_bounds__(256) brick_classify(VmEval ev, Tiles tiles, BrickTask* list, uint32_t* count,
                                                      uint32_t cap, uint32_t* err) {
    brick_classify_body(ev, tiles, list, count, cap, err);
}

template <class Tiles>
__global__ void __launch_bounds__(256) brick_rows(VmEval ev, Tiles tiles, const BrickTask* list,
                                                  const uint32_t* count, uint32_t cap) {
    brick_rows_body(ev, tiles, list, count, cap);
}

// Blocks of a persistent kernel of 256 threads that fill every SM.
inline unsigned persistent_blocks(iso_ctx* ctx, const void* kernel) {
    const int b = resident_blocks(ctx, kernel);
    return (unsigned)((b ? b : 4) * (ctx->sms > 0 ? ctx->sms : 1));
}

// jit.cu: the culled sampler over one lattice with the program's compiled
// evaluator; false (nothing launched) when the program has none
bool jit_sample_bricks(iso_ctx* ctx, const iso_program* prog, const GridTiles& tiles, uint32_t ntiles,
                       BrickTask* list, uint32_t* count, uint32_t cap, cudaError_t* err);

// jit.cu: the full field of one lattice (blocks of eight field_warp warps)
// with the program's compiled evaluator; false (nothing launched) when the
// program has none
bool jit_sample_field(iso_ctx* ctx, const iso_program* prog, const BrickLattice& g, uint64_t blocks,
                      cudaError_t* err);

}  // namespace iso
