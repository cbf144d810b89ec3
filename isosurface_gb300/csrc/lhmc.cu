// LinearHashedMarchingCubes::new(max_depth).extract
// (src/linear_hashed_marching_cubes.rs:62-84) over ImplicitOctree::traverse
// (src/traversal/implicit_octree.rs:39-99) and LinearHashedOctree
// (src/linear_hashed_octree.rs:30-51), with Morton keys (src/morton.rs).
//
// GPU form:
// 1. Octree build in one cooperative launch (oct_build; a launch per
//    generation for long programs and in recordings), generation by
//    generation: evaluate the source
//    at the centres of the children of every refined node, apply
//    should_refine (level < 2 || (level < max_depth && |d| < size * sqrt 3)),
//    and append them in order.  Where a refined node's children go follows
//    from how many nodes before it are refined, which the previous generation
//    left as sums over tiles of nodes; the generations' sizes stay on the
//    device.  Generation g holds keys with 3g+1 bits in ascending order.
// 2. Primal vertices: in the reference every leaf emits primal_vertex(level, i)
//    (morton.rs:120-136) for i < 8; the
//    reference keeps, per vertex, the deepest level (its max-level map).  Of
//    the leaves of that level the one with the smallest key owns the vertex
//    here, which gives a deterministic order (leaf order, then i) for the walk
//    the reference does in HashMap order.  A leaf finds out alone: the cells
//    of its level around the vertex are nodes that are refined (deeper leaves
//    have it), leaves (the smaller key has it) or part of a coarser leaf.
//    That takes the families around: a warp per family of eight children
//    looks up the 27 families around it and tests the family's 27 vertices.
// 3. Dual cubes: for each primal vertex and corner i, the cell dual_vertex(level,
//    REMAP_CUBE[i]) (morton.rs:140-144), or the first of its parents that is a
//    node; the corner is that
//    node's centre and value.  A corner with no ancestor keeps the previous
//    corner's data in the reference (an order-dependent case); it is counted
//    and reported through iso_lhmc_stale_corners.  No input reaches it: all
//    64 level-2 nodes always exist and primal vertices lie strictly inside,
//    so every walk meets a node at level 2 or deeper.  The same warps find
//    them once the vertices before theirs are counted: a corner is a child of
//    one of the 27 families, or the node one of those walks ends at.  The
//    cubes with corners on both sides go to a list, which the later passes
//    walk.
// 4. Marching cubes on the listed cubes with MortonKey dedup: each vertex is
//    owned by the first (cube, first-use rank) that references its key, found
//    with a 64-bit atomicMin in a second hash table.
//
// The host waits twice: for the number of nodes (it sizes the arrays) and for
// the mesh, which is written into the buffers as earlier extractions sized
// them and again where it did not fit.  Every later size is bounded by the
// nodes: splitting a cell adds at most 19 vertices to the octree's 8 nodes,
// so vertices and cubes are below 3 per node.
//
// csg at depth 8 (313 k nodes, 502 k cubes): 690 us with a host round trip
// and three to five launches per generation, hash tables of vertices (128 MB)
// and edges (64 MB) with three lookups per visit, and every pass over all
// cubes.
//
// The reference's output order is that of a RandomState HashMap, so only the
// triangle set (keyed by MortonKey pairs) is defined; this order is
// deterministic.  Keys must fit 31 bits: max_depth <= 10.
#include <cuda_runtime.h>

#include <cstring>

#include <algorithm>
#include <vector>

#include "block_sums.cuh"
#include "internal.h"
#include "vm.cuh"
#define ISO_TABLE static __device__ const
#include "mc_tables.h"

namespace iso {
namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;

// ---------------------------------------------------------------- Morton ---
namespace morton {
constexpr uint64_t DILATE_MASK_2 = 0x7FC0000FF80001FFull;
constexpr uint64_t DILATE_MASK_1 = 0x01C0E070381C0E07ull;
constexpr uint64_t DILATE_MASK_0 = 0x9249249249249249ull;
constexpr uint64_t DILATE_TZ = 0x4924924924924924ull;
constexpr uint64_t DILATE_TY = 0x2492492492492492ull;
constexpr uint64_t DILATE_TX = 0x9249249249249249ull;
constexpr uint64_t DILATE_T1 = 0xB6DB6DB6DB6DB6DBull;
constexpr uint64_t DILATE_T2 = 0xDB6DB6DB6DB6DB6Dull;
constexpr uint64_t DILATE_T3 = 0x6DB6DB6DB6DB6DB6ull;

// morton.rs:54-59 computes floor(ln(k) * 0.48089834696); the constant sits
// just below 1/(3 ln 2), so the result is floor(log2(k) / 3) except at exact
// powers of 8 above 1, where it is one less (checked against the formula for
// every key below 2^31 by the tests).
__host__ __device__ inline int level(uint64_t k) {
    if (k == 0) return 0;
#ifdef __CUDA_ARCH__
    const int msb = 63 - __clzll((long long)k);
#else
    const int msb = 63 - __builtin_clzll(k);
#endif
    int lv = msb / 3;
    if (lv > 0 && k == (1ull << (3 * lv))) lv -= 1;
    return lv;
}
__device__ inline uint64_t parent(uint64_t k) { return max(k >> 3, (uint64_t)1); }
__device__ inline uint64_t add(uint64_t a, uint64_t b) {  // morton.rs:147-157
    return (((a | DILATE_T1) + (b & DILATE_TZ)) & DILATE_TZ) | (((a | DILATE_T2) + (b & DILATE_TY)) & DILATE_TY) |
           (((a | DILATE_T3) + (b & DILATE_TX)) & DILATE_TX);
}
__device__ inline uint64_t sub(uint64_t a, uint64_t b) {  // morton.rs:159-169
    return (((a & DILATE_TZ) - (b & DILATE_TZ)) & DILATE_TZ) | (((a & DILATE_TY) - (b & DILATE_TY)) & DILATE_TY) |
           (((a & DILATE_TX) - (b & DILATE_TX)) & DILATE_TX);
}
__device__ inline V3 center(uint64_t k) {  // morton.rs:78-116
    uint64_t bz = (k >> 2) & DILATE_MASK_0, by = (k >> 1) & DILATE_MASK_0, bx = k & DILATE_MASK_0;
    const int lv = level(k);
    if (lv > 1) {
        bz = (bz | (bz >> 2) | (bz >> 4)) & DILATE_MASK_1;
        by = (by | (by >> 2) | (by >> 4)) & DILATE_MASK_1;
        bx = (bx | (bx >> 2) | (bx >> 4)) & DILATE_MASK_1;
        if (lv > 3) {
            bz = (bz | (bz >> 6) | (bz >> 12)) & DILATE_MASK_2;
            by = (by | (by >> 6) | (by >> 12)) & DILATE_MASK_2;
            bx = (bx | (bx >> 6) | (bx >> 12)) & DILATE_MASK_2;
            if (lv > 9) {
                bz = bz | (bz >> 18) | (bz >> 36);
                by = by | (by >> 18) | (by >> 36);
                bx = bx | (bx >> 18) | (bx >> 36);
            }
        }
    }
    const uint64_t length_mask = (1ull << lv) - 1;
    bz &= length_mask;
    by &= length_mask;
    bx &= length_mask;
    // coordinates are below 2^21: as 32-bit numbers they convert on the FP32
    // side, where 64-bit ones go through the (slow) f64 unit
    const float s = 1.0f / (float)(2u << lv);
    const float s2 = s * 2.0f;
    return v3((float)(uint32_t)bx * s2 + s, (float)(uint32_t)by * s2 + s, (float)(uint32_t)bz * s2 + s);
}
}  // namespace morton

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// open-addressing table of (key, value) slots: key 0 = empty; the slot, or
// NO_SLOT when full
struct alignas(16) Slot {
    unsigned long long key, val;
};
constexpr uint32_t NO_SLOT = 0xFFFFFFFFu;

// The slot of `key`, taken if it has none; *val: a value the slot has held (a
// slot's value only moves one way, so one that `key`'s code cannot improve on
// needs no atomic; neither does a key that is already there).
__device__ __forceinline__ uint32_t ht_insert(Slot* table, uint32_t mask, uint64_t key, unsigned long long* val) {
    uint32_t slot = (uint32_t)mix64(key) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const ulonglong2 q = __ldcg(reinterpret_cast<const ulonglong2*>(table + slot));
        *val = q.y;
        if (q.x == key) return slot;
        if (q.x == 0ull) {
            const unsigned long long prev = atomicCAS(&table[slot].key, 0ull, (unsigned long long)key);
            if (prev == 0ull || prev == key) return slot;
        }
        slot = (slot + 1) & mask;
    }
    return NO_SLOT;
}

// ----------------------------------------------------------- exclusive scan ---
__global__ void __launch_bounds__(1024) scan_blocks(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* sums) {
    __shared__ uint32_t s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * 1024 + threadIdx.x;
    const uint32_t v = i < n ? in[i] : 0u;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) before += s_w[w];
        all += s_w[w];
    }
    if (i < n) out[i] = before + x - v;
    if (threadIdx.x == 0) sums[blockIdx.x] = all;
}

__global__ void __launch_bounds__(1024) scan_sums(uint32_t* sums, uint32_t nb, uint32_t* total) {
    __shared__ uint32_t s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nb; base += 1024) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < nb ? sums[i] : 0u;
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += t;
        }
        if (lane == 31) s_w[warp] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before += s_w[w];
            all += s_w[w];
        }
        if (i < nb) sums[i] = carry + before + x - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void scan_add(uint32_t* out, uint32_t n, const uint32_t* sums) {
    const uint32_t i = blockIdx.x * 1024 + threadIdx.x;
    if (i < n) out[i] += sums[blockIdx.x];
}

// The whole scan in one block for n <= SCAN_SMALL: 16 consecutive entries
// per thread (read before any is written, so in == out is fine).
constexpr uint32_t SCAN_SMALL = 16 * 1024;
__global__ void __launch_bounds__(1024) scan_small(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* total) {
    __shared__ uint32_t s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t i0 = 16 * threadIdx.x;
    uint32_t v[16], sum = 0;
    for (int k = 0; k < 16; ++k) {
        v[k] = i0 + k < n ? in[i0 + k] : 0u;
        sum += v[k];
    }
    uint32_t x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) before += s_w[w];
        all += s_w[w];
    }
    uint32_t run = before + x - sum;
    for (int k = 0; k < 16; ++k) {
        if (i0 + k < n) out[i0 + k] = run;
        run += v[k];
    }
    if (threadIdx.x == 0) *total = all;
}

// ------------------------------------------------------------ octree build ---
constexpr uint32_t TILE = 32;     // nodes with one count of refined ones
constexpr uint32_t OCT_THREADS = 256;
constexpr uint32_t SUPER = 64;    // tiles with one
constexpr uint32_t MAX_GENS = 16; // of any octree (keys fit 31 bits)
constexpr uint32_t BLOCK_FAMILIES = 32;  // families with one sum of primal vertices (block_sums.cuh)
constexpr uint32_t BLOCK_CUBES = 256;    // cubes with one sum of vertices and triangles

// what the passes find out, read back by the host in one copy
struct Ctl {
    uint32_t nodes;
    uint32_t arrived;                       // blocks at the barriers of oct_build
    uint32_t pad[30];
    uint32_t released, pad2;                // turns of the barrier that are over, or ABANDONED (a cache line of its own)
    unsigned long long need;                // nodes the arena had no room for (0: all fit; NO_OCTREE: abandoned)
    unsigned long long work;                // crossing edges of the listed cubes << 32 | listed cubes
    unsigned long long stale;
    uint2 cubes;                            // dual cubes, 0
    uint2 mesh;                             // vertices, triangles
};

constexpr uint32_t ABANDONED = 0xFFFFFFFFu;
constexpr unsigned long long NO_OCTREE = ~0ull;

// One cooperative launch with barriers for programs up to this many ops and
// spheres, a launch per generation beyond and in recordings.  What a block
// waits for at a barrier is the other blocks' evaluations, which have no limit
// of their own (sets of up to 2^24 spheres), while the wait needs one: it ends
// after some seconds, and at the line a generation of 10^9 nodes takes about a
// tenth of one.  A launch is also the faster way where the host's part of it costs
// nothing, as the barriers wait for the slowest block: recorded, a launch per
// generation against one for all, at depth 8: csg 216 and 222 us, a hard set of
// 16 spheres 123 and 128, 64 237 and 250, 256 1115 and 1186, 1023 5673 and
// 6390.  Called without a recording the launches cost 9 us more (csg: 206 and
// 197 us), which they are worth from about 64 spheres on.
constexpr uint64_t BARRIER_COST = 64;

struct OctArgs {
    ProgView pv;
    unsigned long long* keys;  // all nodes, BFS (= ascending) order
    float* vals;
    uint8_t* refine;           // per family (nodes 8 f + 1 .. 8 f + 8): its refined children
    unsigned long long* families;  // refined node's key << 32 | its first child (family_insert)
    uint32_t fmask;
    uint32_t cap;
    uint32_t max_depth;
    uint32_t* tiles;           // refined nodes of every tile, of every super tile: generation g's from
    uint32_t* supers;          // off / TILE + g and off / (TILE * SUPER) + g
    uint2* gens;               // a launch per generation (else null): first node and nodes of generation g
    uint32_t polls;            // limit of a wait
    bool withhold;             // test hook: a block that never comes to the barriers
    Ctl* c;
    Ctl* host;  // page-locked: the size, when it is known
    uint32_t* err;
};

__device__ __forceinline__ bool oct_node(const OctArgs& A, uint32_t at, uint64_t key) {
    const float d = eval_scalar(A.pv, morton::center(key));  // construct_node, implicit_octree.rs:56-59
    const int lv = morton::level(key);
    const float sz = 1.0f / (float)(2u << lv);
    // should_refine (implicit_octree.rs:47-55) with Signed::within_extent (distance.rs:60-62)
    const bool r = lv < 2 || (lv < (int)A.max_depth && fabsf(d) < sz * 1.73205080757f);
    A.keys[at] = key;
    A.vals[at] = d;
    return r;
}

// The nodes by key: a refined node's eight children follow one another in the
// node array, so a table of the refined nodes (0 empty, at most half full)
// finds any node with an eighth of the entries.  A refined node's key fits 32
// bits at the depths allowed.
__device__ __forceinline__ uint32_t family_slot(uint64_t parent, uint32_t mask) {
    const uint32_t h = (uint32_t)parent * 0x9E3779B1u;
    return (h ^ h >> 15) & mask;
}
__device__ __forceinline__ void family_insert(const OctArgs& A, uint64_t parent, uint32_t first, uint32_t slot) {
    for (uint32_t probe = 0; probe <= A.fmask; ++probe, ++slot)
        if (atomicCAS(A.families + (slot & A.fmask), 0ull, parent << 32 | first) == 0ull) return;
}
// the first child of the node with key `parent`, 0 if that is no refined node
__device__ __forceinline__ uint32_t find_family(const unsigned long long* families, uint32_t mask, uint64_t parent) {
    uint32_t slot = family_slot(parent, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long w = __ldg(families + slot);
        if (w == 0ull) return 0;
        if (w >> 32 == parent) return (uint32_t)w;
        slot = (slot + 1) & mask;
    }
    return 0;
}

// All blocks of the (cooperative) launch have come here `turn` times; the
// last one to come releases the others, which wait on a word of its own.
// Bounded: a block whose polls run out marks the count of arrivals.  If the
// turn was not complete then, it is abandoned for all blocks, the last one to
// come among them, which finds the mark; if it was, the mark ends the next
// one.  False, in every thread of every block, once a turn was abandoned.
constexpr uint32_t BARRIER_POLLS = 1u << 22;
constexpr uint32_t GAVE_UP = 1u << 31;
__device__ __forceinline__ bool grid_barrier(const OctArgs& A, uint32_t turn) {
    __shared__ bool s_go;
    __syncthreads();
    if (threadIdx.x == 0) {
        Ctl* c = A.c;
        volatile uint32_t* released = &c->released;
        const uint32_t all = turn * gridDim.x;
        const bool comes = !(A.withhold && blockIdx.x + 1 == gridDim.x);
        uint32_t seen = 0;
        __threadfence();
        const uint32_t before = comes ? atomicAdd(&c->arrived, 1u) : 0u;
        if (before & GAVE_UP) {
            seen = ABANDONED;
        } else if (before + 1 == all) {
            __threadfence();
            *released = seen = turn;
        } else {
            uint32_t polls = 0;
            while ((seen = *released) < turn && ++polls < A.polls) __nanosleep(20);
            if (seen < turn) seen = (atomicOr(&c->arrived, GAVE_UP) & ~GAVE_UP) < all ? ABANDONED : turn;
        }
        if (seen == ABANDONED) {
            *released = ABANDONED;
            atomicOr(A.err, DERR_QUEUE_TIMEOUT);
        }
        __threadfence();
        s_go = seen != ABANDONED;
    }
    __syncthreads();
    return s_go;
}

// Generations first + 1 .. last: the whole octree in one cooperative launch
// (first = 1), a grid barrier between generations, or a launch for each
// generation (A.gens).  Bound by one evaluation's chain per generation: launched
// generation by generation the interpreter's code and the program came from
// L2 again each time (10-18 us each; 95 us for csg at depth 8).
// Generations 0 to 2 (nodes 0, 1-8 and 9-72) every octree has; after that a
// block takes the refined nodes of a tile and evaluates their children.
// What other blocks wrote is read past L1.
__global__ void __launch_bounds__(OCT_THREADS, 4) oct_build(OctArgs A, uint32_t first, uint32_t last) {
    __shared__ unsigned long long s_key[OCT_THREADS];
    __shared__ uint32_t s_sum[OCT_THREADS / 32], s_n[OCT_THREADS / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    auto block_sum = [&](uint32_t v) {
        v = __reduce_add_sync(FULL, v);
        __syncthreads();  // the previous sum and the previous tile are used
        if (lane == 0) s_sum[tid >> 5] = v;
        __syncthreads();
        uint32_t all = 0;
        for (int k = 0; k < OCT_THREADS / 32; ++k) all += s_sum[k];
        return all;
    };
    if (first == 1 && blockIdx.x == 0 && tid < 96) {
        // nodes 1-72 to threads 0-71, so that families are eights of lanes
        const uint32_t at = tid == 72 ? 0 : tid + 1;
        bool r = false;
        if (tid <= 72) r = oct_node(A, at, at == 0 ? 1 : at < 9 ? 7 + at : 55 + at);
        const uint32_t m = __ballot_sync(FULL, r) >> (lane & ~7u) & 0xFFu;
        if (tid < 72 && (tid & 7) == 0) {
            A.refine[at >> 3] = (uint8_t)m;
            family_insert(A, at == 1 ? 1 : 7 + (at >> 3), at, family_slot(at == 1 ? 1 : 7 + (at >> 3), A.fmask));
            if (at >= 9) {
                atomicAdd(A.tiles + 9 / TILE + 2 + (at - 9) / TILE, (uint32_t)__popc(m));
                atomicAdd(A.supers + 9 / (TILE * SUPER) + 2, (uint32_t)__popc(m));
            }
        }
    }
    uint32_t off = 9, cnt = 64;
    unsigned long long need = 0;
    if (first > 2) {
        const uint2 gen = A.gens[first];
        off = gen.x;
        cnt = gen.y;
        if (cnt == 0) return;  // the build is over
    }
    for (uint32_t g = max(first, 2u); g < last; ++g) {
        if (!A.gens && !grid_barrier(A, g - 1)) {
            if (blockIdx.x == 0 && tid == 0) {
                A.host->need = NO_OCTREE;
            }
            return;
        }
        const uint32_t next = off + cnt;
        const uint32_t ntiles = (cnt + TILE - 1) / TILE, nsupers = (ntiles + SUPER - 1) / SUPER;
        const uint32_t* tiles = A.tiles + off / TILE + g;
        const uint32_t* supers = A.supers + off / (TILE * SUPER) + g;
        uint32_t* ntile = A.tiles + next / TILE + g + 1;
        uint32_t* nsuper = A.supers + next / (TILE * SUPER) + g + 1;
        // tiles a block takes together: one while there are blocks for all, up
        // to a node per thread, so that a block's chain of loads and its lanes'
        // last evaluation are paid for once
        const uint32_t span = min((ntiles + gridDim.x - 1) / gridDim.x, OCT_THREADS / TILE);
        for (uint32_t t = blockIdx.x * span; t < ntiles; t += gridDim.x * span) {
            const uint32_t s = t / SUPER;
            uint32_t sum = 0;
            for (uint32_t k = tid; k < s; k += OCT_THREADS) sum += __ldcg(supers + k);
            for (uint32_t k = s * SUPER + tid; k < t; k += OCT_THREADS) sum += __ldcg(tiles + k);
            // its nodes and which of them are refined (on their way meanwhile)
            const uint32_t i = t * TILE + tid, at = off + i;  // node 8 f + 1 + bit
            const bool mine = tid < span * TILE && i < cnt;
            const uint32_t flags = mine ? __ldcg(A.refine + ((at - 1) >> 3)) : 0u;
            const unsigned long long node = mine ? __ldcg(A.keys + at) : 0ull;
            const uint32_t before = block_sum(sum);
            // the refined ones, in order
            const bool r = flags >> ((at - 1) & 7) & 1;
            const uint32_t m = __ballot_sync(FULL, r);
            if (lane == 0) s_n[tid >> 5] = __popc(m);
            __syncthreads();
            uint32_t n = 0;
            for (uint32_t w = 0; w < OCT_THREADS / 32; ++w) {
                if (r && w == tid >> 5) s_key[n + __popc(m & ((1u << lane) - 1u))] = node;
                n += s_n[w];
            }
            n *= 8;
            __syncthreads();
            for (uint32_t c0 = 0; c0 < n; c0 += OCT_THREADS) {
                const uint32_t c = c0 + tid, rel = 8 * before + c;
                const bool live = c < n && next + rel < A.cap, leads = live && (lane & 7) == 0;
                const unsigned long long parent = c < n ? s_key[c >> 3] : 0ull;
                // the family's place in the table is asked for before the evaluation
                uint32_t slot = family_slot(parent, A.fmask);
                unsigned long long taken = 0;
                if (leads) taken = atomicCAS(A.families + slot, 0ull, parent << 32 | (next + rel));
                bool cr = false;
                if (live) cr = oct_node(A, next + rel, parent << 3 | (c & 7));  // Morton::child
                const uint32_t cm = __ballot_sync(FULL, cr) >> (lane & ~7u) & 0xFFu;
                if (leads) {  // a family lies in one tile
                    if (taken) family_insert(A, parent, next + rel, slot + 1);
                    A.refine[(next + rel) >> 3] = (uint8_t)cm;
                    if (cm) {
                        atomicAdd(ntile + rel / TILE, (uint32_t)__popc(cm));
                        atomicAdd(nsuper + rel / (TILE * SUPER), (uint32_t)__popc(cm));
                    }
                }
            }
        }
        // the next generation's size, in every block
        uint32_t sum = 0;
        for (uint32_t k = tid; k < nsupers; k += OCT_THREADS) sum += __ldcg(supers + k);
        const uint64_t children = 8ull * block_sum(sum);
        const bool fits = next + children <= A.cap;
        off = next;
        cnt = fits ? (uint32_t)children : 0u;
        if (cnt == 0) {
            if (!fits) need = next + children;
            break;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        A.c->nodes = A.host->nodes = off + cnt;
        A.c->need = A.host->need = need;
        if (A.gens) A.gens[last] = make_uint2(off, cnt);
    }
}

// ---------------------------------------------------------------- dual cubes ---
struct CubeArgs {
    const unsigned long long* nkeys;
    const float* nvals;
    const uint8_t* refine;
    const unsigned long long* families;
    uint32_t fmask;
    uint32_t nfamilies;
    uint8_t* fcount;         // per family: primal vertices its children own
    unsigned long long* fsums;  // per BLOCK_FAMILIES families
    uint32_t cap;            // room for cubes
    Ctl* c;
    uint8_t* cases;          // per cube
    uint2* list;             // listed cubes (both kinds of corners): cube, case
    uint32_t* corner;        // 8 node indices per listed cube (UINT32_MAX: no ancestor)
    uint32_t* slots;         // 12 per listed cube: the slots of its edges' keys, by first-use rank
    Slot* table;             // edge key -> first visitor: cube << 4 | first-use rank
    uint32_t table_cap;
    uint16_t* owned;         // per cube: owned first-use ranks
    unsigned long long* sums;  // per BLOCK_CUBES cubes: triangles << 32 | vertices
    uint32_t *vbase, *tbase;   // per cube, of the listed ones
    float* out_v;
    uint32_t* out_i;
    uint64_t* out_k;
    uint32_t cap_v, cap_t;
    uint32_t* err;
    Ctl* host;           // page-locked: the counters and the error flags at the end
    uint64_t* host_err;
};

// What a warp knows of family f (first child 8 f + 1) and its surroundings:
// lane n < 27 looks after the family at offset (n % 3, n / 3 % 3, n / 9) - 1
// and the vertex at that offset (0..2 per axis, in children's sizes).
struct Around {
    uint32_t first;  // that family's first child, 0: none
    uint32_t refine; // its refined children
    uint64_t key;    // its parent's key
    bool own;        // a child of this family owns the lane's vertex
    uint32_t code;   // child * 8 + vertex of it
    uint32_t lo, hi; // the set of all such codes (in every lane)
};

// the cells around vertex offset v on one axis: cell a = 0 (below), 1 (above)
// is child bit `bit` of the family at offset `fam`
__device__ __forceinline__ uint32_t axis_fam(uint32_t v, uint32_t a) { return (v + 1 + a) >> 1; }
__device__ __forceinline__ uint32_t axis_bit(uint32_t v, uint32_t a) { return (v + 1 + a) & 1; }

__device__ __forceinline__ Around look_around(const CubeArgs& A, uint32_t f) {
    const uint32_t lane = threadIdx.x & 31, n = min(lane, 26u);
    const uint32_t vx = n % 3, vy = n / 3 % 3, vz = n / 9;
    const uint64_t P = __ldg(A.nkeys + 8 * f + 1) >> 3;
    const int L = (63 - __clzll((long long)P)) / 3;
    Around q;
    // (P - (1, 1, 1)) + offset, per axis; past the domain's faces this is some
    // other key, which only a vertex on the face would look at
    q.key = morton::add(morton::sub(P, 7), (uint64_t)((vx & 1) | (vx >> 1) << 3 | (vy & 1) << 1 | (vy >> 1) << 4 |
                                                       (vz & 1) << 2 | (vz >> 1) << 5));
    q.first = n == 13 ? 8 * f + 1 : find_family(A.families, A.fmask, q.key);
    q.refine = q.first ? __ldg(A.refine + (q.first >> 3)) : 0u;
    // strictly inside the domain (morton.rs:120-136)
    const uint64_t lead = 1ull << (3 * L), low = P ^ lead;
    auto inside = [&](uint32_t v, uint64_t axis) {
        const uint64_t all = axis & (lead - 1), at = low & axis;
        return !(v == 0 && at == 0) && !(v == 2 && at == all);
    };
    bool own = lane < 27 && inside(vx, morton::DILATE_TX) && inside(vy, morton::DILATE_TY) && inside(vz, morton::DILATE_TZ);
    uint64_t least = ~0ull;
    uint32_t mine = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t a = k & 1, b = k >> 1 & 1, c = k >> 2;
        const uint32_t from = axis_fam(vx, a) + 3 * axis_fam(vy, b) + 9 * axis_fam(vz, c);
        const uint32_t ci = axis_bit(vx, a) | axis_bit(vy, b) << 1 | axis_bit(vz, c) << 2;
        const uint32_t word = __shfl_sync(FULL, q.refine | (q.first ? 256u : 0u), from);
        const uint64_t key = (uint64_t)__shfl_sync(FULL, (uint32_t)q.key, from) << 3 | ci;
        if (!(word & 256u)) continue;  // a coarser leaf's
        if (word >> ci & 1u) own = false;
        // key 8^lv has one level less by morton::level, and no vertices
        if (key < least && key != lead << 3) {
            least = key;
            mine = from == 13 ? ci + 1 : 0;
        }
    }
    q.own = own && mine;
    const uint32_t child = mine - 1;
    q.code = 8 * child + ((vx - (child & 1)) | (vy - (child >> 1 & 1)) << 1 | (vz - (child >> 2)) << 2);
    q.lo = __reduce_or_sync(FULL, q.own && q.code < 32 ? 1u << q.code : 0u);
    q.hi = __reduce_or_sync(FULL, q.own && q.code >= 32 ? 1u << (q.code - 32) : 0u);
    return q;
}

// Primal vertices of every family: a warp each, a block's 8 warps over
// BLOCK_FAMILIES.  (A hash table of vertices with an insertion per leaf and
// corner and two lookups took 41 + 31 + 33 us for 313 k nodes, a lane per
// leaf and corner with its seven lookups 72.)
__global__ void __launch_bounds__(256) family_count(CubeArgs A) {
    __shared__ uint32_t s_n[8];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t n = 0;
    for (uint32_t k = warp; k < BLOCK_FAMILIES; k += 8) {
        const uint32_t f = blockIdx.x * BLOCK_FAMILIES + k;
        if (f >= A.nfamilies) break;
        const Around q = look_around(A, f);
        const uint32_t own = __popc(q.lo) + __popc(q.hi);
        if (lane == 0) A.fcount[f] = (uint8_t)own;
        n += own;
    }
    if (lane == 0) s_n[warp] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
        for (int w = 0; w < 8; ++w) all += s_n[w];
        A.fsums[blockIdx.x] = all;
    }
}

// The dual cubes of the families' vertices (in order of leaf, then vertex):
// corners, case, and the list of those with corners on both sides, with one
// place in it for a block's eight families (one for every warp's cubes, all
// at one address, cost more than the walks).
__global__ void __launch_bounds__(256) cube_gather(CubeArgs A) {
    __shared__ uint32_t s_listed[8], s_edges[8], s_base;
    const unsigned long long base = A.fsums[blockIdx.x];
    if (base == NO_ITEMS) return;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, f0 = blockIdx.x * BLOCK_FAMILIES;
    // vertices before each of the block's families (lane = family)
    const uint32_t count = f0 + lane < A.nfamilies ? A.fcount[f0 + lane] : 0u;
    uint32_t before = count;
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(FULL, before, o);
        if (lane >= o) before += up;
    }
    before += (uint32_t)base - count;
    for (uint32_t k = warp; k < BLOCK_FAMILIES; k += 8) {
        const uint32_t f = f0 + k, n = __shfl_sync(FULL, count, k), j0 = __shfl_sync(FULL, before, k);
        bool listed = false;
        uint32_t corner[8], cs = 0, j = 0;
        if (n) {  // warp-uniform
            Around q = look_around(A, f);
            // where there is no family, or its children's keys are past 32
            // bits, the walk goes on at its parent
            uint32_t ref = q.first;
            if (lane < 27 && (!q.first || q.key >> 29)) {
                uint64_t m = q.key;
                uint32_t found = 0xFFFFFFFFu;
                while (m > 1) {
                    const uint32_t g = m >> 32 ? 0u : find_family(A.families, A.fmask, m >> 3);
                    if (g) {
                        found = g + (uint32_t)(m & 7);
                        break;
                    }
                    m = morton::parent(m);
                }
                ref = found;
                q.first = 0;
            }
            const uint32_t vx = min(lane, 26u) % 3, vy = min(lane, 26u) / 3 % 3, vz = min(lane, 26u) / 9;
            uint32_t prev = 0xFFFFFFFFu;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                constexpr uint8_t REMAP[8] = {2, 3, 1, 0, 6, 7, 5, 4};  // iso_remap_cube: vertex - REMAP = cell
                const uint32_t a = ~REMAP[i] & 1, b = ~REMAP[i] >> 1 & 1, c = ~REMAP[i] >> 2 & 1;
                const uint32_t from = axis_fam(vx, a) + 3 * axis_fam(vy, b) + 9 * axis_fam(vz, c);
                const uint32_t ci = axis_bit(vx, a) | axis_bit(vy, b) << 1 | axis_bit(vz, c) << 2;
                uint32_t found = __shfl_sync(FULL, ref, from);
                if (__shfl_sync(FULL, q.first, from)) found += ci;
                if (q.own && found == 0xFFFFFFFFu) {
                    // the reference keeps the previous corner's data here (implicit_octree.rs:84-95)
                    atomicAdd(&A.c->stale, 1ull);
                    found = prev;
                }
                corner[i] = found;
                prev = found;
            }
            if (q.own) {
                const unsigned long long set = (unsigned long long)q.hi << 32 | q.lo;
                j = j0 + __popcll(set & ((1ull << q.code) - 1));
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const float d = corner[i] != 0xFFFFFFFFu ? __ldg(A.nvals + corner[i]) : 0.0f;
                    if (!(d > 0.0f)) cs |= 1u << i;
                }
                if (j < A.cap) A.cases[j] = (uint8_t)cs;
                else atomicOr(A.err, DERR_CAPACITY);
                listed = j < A.cap && cs != 0 && cs != 255;
            }
        }
        const uint32_t lm = __ballot_sync(FULL, listed);
        const uint32_t edges = __reduce_add_sync(FULL, listed ? (uint32_t)iso_edge_count[cs] : 0u);
        if (lane == 0) {
            s_listed[warp] = __popc(lm);
            s_edges[warp] = edges;
        }
        __syncthreads();
        uint32_t at = 0, all = 0, ne = 0;
        for (uint32_t w = 0; w < 8; ++w) {
            if (w < warp) at += s_listed[w];
            all += s_listed[w];
            ne += s_edges[w];
        }
        if (threadIdx.x == 0 && all)
            s_base = (uint32_t)atomicAdd(&A.c->work, (unsigned long long)ne << 32 | (unsigned long long)all);
        __syncthreads();
        if (listed) {
            at += s_base + __popc(lm & ((1u << lane) - 1u));
            A.list[at] = make_uint2(j, cs);
            uint4* c = reinterpret_cast<uint4*>(A.corner + 8 * (size_t)at);
            c[0] = make_uint4(corner[0], corner[1], corner[2], corner[3]);
            c[1] = make_uint4(corner[4], corner[5], corner[6], corner[7]);
        }
        __syncthreads();  // s_base and s_listed are used
    }
}

// the edge table's mask: three slots for every two crossing edges of listed
// cubes (an edge has about four cubes), as far as there is room
__device__ __forceinline__ uint32_t edge_mask(const CubeArgs& A) {
    const uint32_t visits = (uint32_t)(A.c->work >> 32), want = max(visits + visits / 2, 1024u);
    const uint32_t bits = 32 - __clz(want - 1);
    return min(bits >= 31 ? 1u << 31 : 1u << bits, A.table_cap) - 1;
}

__global__ void __launch_bounds__(256) edge_clear(CubeArgs A) {
    const uint32_t mask = edge_mask(A);
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i <= mask; i += gridDim.x * 256)
        reinterpret_cast<ulonglong2*>(A.table)[i] = make_ulonglong2(0ull, ~0ull);
}

__device__ __forceinline__ uint64_t edge_key(const unsigned long long* nkeys, const uint32_t* corner, uint32_t e) {
    const uint32_t u = corner[iso_edge_connection[e][0]], w = corner[iso_edge_connection[e][1]];
    const uint64_t a = u != 0xFFFFFFFFu ? nkeys[u] : 1ull, b = w != 0xFFFFFFFFu ? nkeys[w] : 1ull;
    return a > b ? ((b << 32) | a) : ((a << 32) | b);  // MortonKey::new, index_cache.rs:63-73
}

// in the table an edge goes by its two nodes, as its keys do one by one
// (+ 1: never 0)
__device__ __forceinline__ uint64_t edge_nodes(const uint32_t* corner, uint32_t e) {
    const uint32_t u = corner[iso_edge_connection[e][0]], w = corner[iso_edge_connection[e][1]];
    const uint32_t a = u != 0xFFFFFFFFu ? u : 0u, b = w != 0xFFFFFFFFu ? w : 0u;  // node 0 has key 1
    return (a > b ? (uint64_t)b << 32 | a : (uint64_t)a << 32 | b) + 1;
}

// Four lanes per cube: a visit is a chain of dependent accesses to L2.
__global__ void __launch_bounds__(256) edge_visit(CubeArgs A) {
    const uint32_t n = (uint32_t)A.c->work, mask = edge_mask(A), sub = threadIdx.x & 3;
    for (uint32_t p = blockIdx.x * 64 + (threadIdx.x >> 2); p < n; p += gridDim.x * 64) {
        const uint2 q = A.list[p];
        const uint64_t ord = iso_edge_order[q.y];
        const uint32_t ne = iso_edge_count[q.y];
        for (uint32_t r = sub; r < ne; r += 4) {
            const uint32_t e = (uint32_t)(ord >> (4 * r)) & 15u;
            const unsigned long long code = (unsigned long long)q.x << 4 | r;
            unsigned long long held;
            const uint32_t slot = ht_insert(A.table, mask, edge_nodes(A.corner + 8 * (size_t)p, e), &held);
            A.slots[12 * (size_t)p + r] = slot;
            if (slot == NO_SLOT) atomicOr(A.err, DERR_CAPACITY);
            else if (held > code) atomicMin(&A.table[slot].val, code);
        }
    }
}

__global__ void __launch_bounds__(128) edge_own(CubeArgs A) {
    const uint32_t n = (uint32_t)A.c->work, lane = threadIdx.x & 31;
    for (uint32_t p0 = blockIdx.x * 128 + (threadIdx.x & ~31u); p0 < n; p0 += gridDim.x * 128) {
        const uint32_t p = p0 + lane;
        const uint2 q = p < n ? A.list[p] : make_uint2(0, 0);
        const uint32_t ne = iso_edge_count[q.y];
        uint32_t own = 0;
        for (uint32_t r = 0; r < ne; ++r) {
            const uint32_t slot = A.slots[12 * (size_t)p + r];
            if (slot != NO_SLOT && A.table[slot].val == (((uint64_t)q.x << 4) | r)) own |= 1u << r;
        }
        if (p < n) A.owned[q.x] = (uint16_t)own;
        // the list keeps a block's cubes together, so a warp mostly adds to one sum
        const uint32_t b = q.x / BLOCK_CUBES, b0 = __shfl_sync(FULL, b, 0);
        const bool same = p < n && b == b0;
        const uint32_t nv = __popc(own), nt = iso_tri_count[q.y];
        const uint32_t sv = __reduce_add_sync(FULL, same ? nv : 0u), st = __reduce_add_sync(FULL, same ? nt : 0u);
        if (lane == 0) atomicAdd(A.sums + b0, (unsigned long long)st << 32 | (unsigned long long)sv);
        else if (p < n && !same) atomicAdd(A.sums + b, (unsigned long long)nt << 32 | (unsigned long long)nv);
    }
}

// a thread block per BLOCK_CUBES cubes, a thread per cube
__global__ void __launch_bounds__(256) cube_offsets(CubeArgs A) {
    const unsigned long long base = A.sums[blockIdx.x];
    if (base == NO_ITEMS) return;
    const uint32_t n = min(A.c->cubes.x, A.cap), j = blockIdx.x * BLOCK_CUBES + threadIdx.x;
    const uint32_t cs = j < n ? A.cases[j] : 0u;
    const bool listed = cs != 0 && cs != 255;
    const unsigned long long mine =
        listed ? (unsigned long long)iso_tri_count[cs] << 32 | (unsigned long long)__popc(A.owned[j]) : 0ull;
    const unsigned long long run = offset_in_block(base, mine);
    if (listed) {
        A.vbase[j] = (uint32_t)run;
        A.tbase[j] = (uint32_t)(run >> 32);
    }
}

__global__ void __launch_bounds__(128) cube_emit(CubeArgs A) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // all final by now
        *A.host = *A.c;
        *A.host_err = *A.err;
    }
    const uint32_t n = (uint32_t)A.c->work;
    for (uint32_t p = blockIdx.x * 128 + threadIdx.x; p < n; p += gridDim.x * 128) {
        const uint2 q = A.list[p];
        const uint32_t j = q.x, cs = q.y, nt = iso_tri_count[cs], ne = iso_edge_count[cs];
        const uint32_t* corner = A.corner + 8 * (size_t)p;
        const uint64_t ord = iso_edge_order[cs];
        const uint32_t own = A.owned[j], vb = A.vbase[j];
        uint32_t ids[12];
        for (uint32_t r = 0; r < ne; ++r) {
            if ((own >> r) & 1u) {
                const uint32_t e = (uint32_t)(ord >> (4 * r)) & 15u;
                const uint32_t vid = vb + __popc(own & ((1u << r) - 1u));
                ids[r] = vid;
                if (vid >= A.cap_v) continue;
                // find_crossing_point over the two corner nodes (distance.rs:64-69)
                const uint32_t u = corner[iso_edge_connection[e][0]], w = corner[iso_edge_connection[e][1]];
                const uint64_t ku = u != 0xFFFFFFFFu ? A.nkeys[u] : 1ull, kw = w != 0xFFFFFFFFu ? A.nkeys[w] : 1ull;
                const float fa = u != 0xFFFFFFFFu ? A.nvals[u] : 0.0f, fb = w != 0xFFFFFFFFu ? A.nvals[w] : 0.0f;
                const V3 pa = morton::center(ku), pb = morton::center(kw);
                const float delta = fb - fa;
                const float t = (delta == 0.0f) ? 0.5f : -fa / delta;
                const float omt = 1.0f - t;
                A.out_v[3 * (size_t)vid + 0] = pa.x * omt + pb.x * t;
                A.out_v[3 * (size_t)vid + 1] = pa.y * omt + pb.y * t;
                A.out_v[3 * (size_t)vid + 2] = pa.z * omt + pb.z * t;
                if (A.out_k) {
                    const uint64_t k = edge_key(A.nkeys, corner, e);
                    A.out_k[2 * (size_t)vid] = k >> 32;
                    A.out_k[2 * (size_t)vid + 1] = k & 0xFFFFFFFFull;
                }
            } else {
                const uint32_t slot = A.slots[12 * (size_t)p + r];
                ids[r] = 0;
                if (slot == NO_SLOT) continue;  // reported when it found no room
                const uint64_t code = A.table[slot].val;
                const uint32_t oj = (uint32_t)(code >> 4), orank = (uint32_t)(code & 15u);
                ids[r] = A.vbase[oj] + __popc((uint32_t)A.owned[oj] & ((1u << orank) - 1u));
            }
        }
        const uint64_t slotw = iso_tri_slot[cs];
        const uint32_t t0 = A.tbase[j];
        for (uint32_t k = 0; k < 3 * nt; ++k)
            if (t0 + k / 3 < A.cap_t) A.out_i[3 * (size_t)t0 + k] = ids[(slotw >> (4 * k)) & 15u];
    }
}

}  // namespace

// exclusive scan of n u32 into out; sums needs (n + 1023) / 1024 entries
iso_status scan_u32(iso_ctx* ctx, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* sums, uint32_t* total) {
    const uint32_t nb = (n + 1023) / 1024;
    if (n == 0) {
        cudaMemsetAsync(total, 0, 4, ctx->stream);
        return ISO_OK;
    }
    if (n <= SCAN_SMALL) {
        scan_small<<<1, 1024, 0, ctx->stream>>>(in, out, n, total);
        ctx->launches++;
        return check_launch(ctx, "scan");
    }
    scan_blocks<<<nb, 1024, 0, ctx->stream>>>(in, out, n, sums);
    scan_sums<<<1, 1024, 0, ctx->stream>>>(sums, nb, total);
    scan_add<<<nb, 1024, 0, ctx->stream>>>(out, n, sums);
    ctx->launches += 3;
    return check_launch(ctx, "scan");
}

}  // namespace iso

using namespace iso;

namespace {

struct Arena {
    char* base;
    size_t used, cap;
    template <class T>
    T* take(size_t n) {
        size_t at = (used + 255) & ~(size_t)255;
        used = at + n * sizeof(T);
        return used <= cap ? reinterpret_cast<T*>(base + at) : nullptr;
    }
};

uint32_t pow2_at_least(uint64_t v) {
    uint64_t p = 1024;
    while (p < v) p <<= 1;
    return (uint32_t)std::min<uint64_t>(p, 1ull << 31);
}

unsigned blocks_for(const iso_ctx* ctx, uint64_t items, unsigned per_block, unsigned per_sm) {
    const uint64_t want = (items + per_block - 1) / per_block;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)std::max(ctx->sms, 1) * per_sm));
}

}  // namespace

// The counts an extraction discovered: its nodes, dual cubes, triangles and
// vertices.  An eager run fills one; a run recorded into a CUDA graph replays
// one (queueing everything, synchronising nowhere); its kernels store each
// count in pinned memory, so that the replay can be checked against the trace.
struct LhmcTrace {
    uint32_t nodes = 0, ncubes = 0, nt = 0, nv = 0;
};
// h_pinned slots: [3] error flags, [8 ..] the device counters
constexpr int LHMC_PIN_CTL = 8;
static_assert(8 * LHMC_PIN_CTL + sizeof(Ctl) <= 4096, "pinned scratch");

static LhmcTrace counts_of(const iso_ctx* ctx) {
    const Ctl* c = (const Ctl*)(ctx->h_pinned + LHMC_PIN_CTL);
    return LhmcTrace{c->nodes, c->cubes.x, c->mesh.y, c->mesh.x};
}

// blocks of oct_build, all of which are resident at once
static unsigned oct_blocks(iso_ctx* ctx) {
    static_assert(OCT_THREADS == 256, "resident_blocks");
    const int b = std::max(1, std::min(resident_blocks(ctx, (const void*)oct_build), 4));
    return (unsigned)(b * std::max(ctx->sms, 1));
}

static iso_status lhmc_extract_impl(iso_ctx* ctx, const iso_program* prog, uint32_t max_depth, uint32_t flags,
                                       iso_mesh_info* info, LhmcTrace* trace, const LhmcTrace* replay) {
    if (!ctx || !prog) return ISO_ERR_INVALID_ARG;
    if (prog->ctx != ctx) return fail(ctx, ISO_ERR_INVALID_ARG, "program belongs to another context");
    if (max_depth > 10) return fail(ctx, ISO_ERR_INVALID_ARG, "max_depth above 10 (Morton keys must fit 31 bits)");
    if (flags & ~(uint32_t)ISO_FLAG_KEYS) return fail(ctx, ISO_ERR_INVALID_ARG, "unsupported flags");
    iso_status s = set_device(ctx);
    if (s != ISO_OK) return s;
    const bool rec = replay != nullptr;
    if (!rec) {
        ctx->last = iso_mesh_info{};
        ctx->last_flags = flags;
        ctx->last_vertex_floats = 3;
    }
    StageTimer timer(ctx, ISO_STAGE_OCTREE);
    // ---- 1. octree, generation by generation (root, then 8 per refined node)
    uint64_t max_nodes = 1;
    {
        uint64_t gen = 1;
        for (uint32_t g = 0; g < max_depth + 2; ++g) {
            gen *= 8;
            max_nodes += gen;
            if (max_nodes > (1ull << 28)) break;
        }
    }
    // counters, generations, tile counts and the table of families | keys | values | refine flags
    auto tile_words = [](size_t cap) { return 2 * MAX_GENS + cap / TILE + cap / (TILE * SUPER) + 3 * MAX_GENS; };
    auto table_at = [&](size_t cap) { return (sizeof(Ctl) + 4 * tile_words(cap) + 255) & ~(size_t)255; };
    auto head_bytes = [&](size_t cap) { return table_at(cap) + 8 * (size_t)pow2_at_least(cap / 4); };
    auto node_bytes = [&](size_t cap) { return head_bytes(cap) + 12 * cap + cap / 8 + 4096; };
    // a first guess, or what this octree had last time: the arena may be larger
    // from other ones, but the table in it is cleared for each build
    uint64_t guess = 1ull << 20;
    for (const auto& r : ctx->lhmc_rooms)
        if (r.program == prog->content_hash && r.depth == max_depth) guess = std::max(guess, r.nodes);
    size_t node_cap = (size_t)std::min(max_nodes, guess);
    const uint32_t last = std::max(2u, max_depth) + 1;  // the last generation there can be: see morton::level
    Ctl* const h = (Ctl*)(ctx->h_pinned + LHMC_PIN_CTL);
    cudaError_t e;
    OctArgs oa{};
    uint32_t nodes = 0;
    while (true) {
        if ((s = ensure(ctx, ctx->aux, node_bytes(node_cap))) != ISO_OK) return s;
        Arena a{(char*)ctx->aux.p, 0, ctx->aux.bytes};
        char* head = a.take<char>(head_bytes(node_cap));
        oa.pv = prog->view();
        oa.keys = a.take<unsigned long long>(node_cap);
        oa.vals = a.take<float>(node_cap);
        oa.refine = a.take<uint8_t>(node_cap / 8 + 1);
        oa.families = (unsigned long long*)(head + table_at(node_cap));
        oa.fmask = pow2_at_least(node_cap / 4) - 1;
        oa.cap = (uint32_t)node_cap;
        oa.max_depth = max_depth;
        oa.c = (Ctl*)head;
        oa.host = h;
        oa.err = ctx->d_err;
        uint2* gens = (uint2*)(oa.c + 1);
        oa.tiles = (uint32_t*)(gens + MAX_GENS);
        oa.supers = oa.tiles + node_cap / TILE + MAX_GENS;
        e = cudaMemsetAsync(head, 0, head_bytes(node_cap), ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "octree counters");
        // blocks beyond the widest generation's tiles would only come to the barriers
        const uint64_t most = std::min<uint64_t>(1ull << std::min(3 * (last - 1), 32u), node_cap);
        const unsigned blocks = (unsigned)std::min<uint64_t>(oct_blocks(ctx), (most + TILE - 1) / TILE);
        if (prog->cost <= BARRIER_COST && !rec) {
            oa.withhold = debug_waits_run_out();
            oa.polls = oa.withhold ? 256 : BARRIER_POLLS;
            uint32_t first_arg = 1, last_arg = last;
            void* args[] = {&oa, &first_arg, &last_arg};
            e = cudaLaunchCooperativeKernel(oct_build, dim3(blocks), dim3(OCT_THREADS), args, 0, ctx->stream);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "octree launch");
            ctx->launches++;
        } else {
            oa.gens = gens;
            for (uint32_t g = 1; g < last; ++g) {
                oct_build<<<g == 1 ? 1 : blocks, OCT_THREADS, 0, ctx->stream>>>(oa, g, g + 1);
                ctx->launches++;
            }
        }
        if ((s = check_launch(ctx, "octree")) != ISO_OK) return s;
        if (rec) {
            nodes = replay->nodes;
            break;
        }
        e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "read octree size");
        if (h->need == NO_OCTREE) {
            s = read_device_errors(ctx);
            return s != ISO_OK ? s : fail(ctx, ISO_ERR_TIMEOUT, "octree barrier gave up");
        }
        if (h->need == 0) {
            nodes = h->nodes;
            if (nodes > guess)
                ctx->lhmc_rooms[ctx->lhmc_next_room++ % 8] = iso_ctx::OctreeRoom{prog->content_hash, max_depth, nodes};
            break;
        }
        // a generation did not fit: again in a larger arena
        if (h->need >= 0xFFFFFFF0ull) return fail(ctx, ISO_ERR_TOO_LARGE, "octree too large");
        node_cap = (size_t)std::max<uint64_t>(h->need, std::min<uint64_t>(2 * (uint64_t)node_cap, 0xFFFFFFF0ull));
    }
    if (trace) trace->nodes = nodes;

    // ---- 2. to 4. primal vertices, dual cubes and their marching cubes
    const uint64_t bound = 3ull * nodes + 1024;  // vertices, and the dual cubes around them
    const uint32_t nfam = (nodes - 1) / 8;
    const uint32_t fblocks = (nfam + BLOCK_FAMILIES - 1) / BLOCK_FAMILIES;
    const uint32_t cblocks = (uint32_t)((bound + BLOCK_CUBES - 1) / BLOCK_CUBES);
    if ((s = ensure(ctx, ctx->aux2, 8ull * (fblocks + cblocks) + nfam + 4096)) != ISO_OK) return s;
    const uint32_t ecap = pow2_at_least(4 * bound);
    if ((s = ensure(ctx, ctx->aux3, (32ull + 8 + 48 + 1 + 2 + 8) * bound + 16ull * ecap + 8192)) != ISO_OK) return s;
    // a first extraction starts from a modest guess; later ones reuse what grew
    const bool keys = (flags & ISO_FLAG_KEYS) != 0;
    if ((s = ensure(ctx, ctx->mesh_v, 12 * (size_t)65536)) != ISO_OK) return s;
    if ((s = ensure(ctx, ctx->mesh_i, 12 * (size_t)131072)) != ISO_OK) return s;
    if (keys && (s = ensure(ctx, ctx->mesh_k, 16 * (size_t)65536)) != ISO_OK) return s;
    Arena a3{(char*)ctx->aux3.p, 0, ctx->aux3.bytes};
    Arena a2{(char*)ctx->aux2.p, 0, ctx->aux2.bytes};
    CubeArgs ca{};
    ca.nkeys = oa.keys;
    ca.nvals = oa.vals;
    ca.refine = oa.refine;
    ca.families = oa.families;
    ca.fmask = oa.fmask;
    ca.nfamilies = nfam;
    ca.fsums = a2.take<unsigned long long>(fblocks);
    ca.sums = a2.take<unsigned long long>(cblocks);
    ca.fcount = a2.take<uint8_t>(nfam);
    ca.cap = (uint32_t)bound;
    ca.c = oa.c;
    ca.table = a3.take<Slot>(ecap);
    ca.table_cap = ecap;
    ca.corner = a3.take<uint32_t>(8 * bound);
    ca.list = a3.take<uint2>(bound);
    ca.slots = a3.take<uint32_t>(12 * bound);
    ca.cases = a3.take<uint8_t>(bound);
    ca.owned = a3.take<uint16_t>(bound);
    ca.vbase = a3.take<uint32_t>(bound);
    ca.tbase = a3.take<uint32_t>(bound);
    ca.err = ctx->d_err;
    ca.host = h;
    ca.host_err = ctx->h_pinned + 3;
    e = cudaMemsetAsync(ca.sums, 0, 8ull * cblocks, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "clear sums");
    family_count<<<fblocks, 256, 0, ctx->stream>>>(ca);
    scan_block_sums<<<1, 1024, 0, ctx->stream>>>(ca.fsums, fblocks, &oa.c->cubes);
    cube_gather<<<fblocks, 256, 0, ctx->stream>>>(ca);
    edge_clear<<<blocks_for(ctx, ecap, 256, 8), 256, 0, ctx->stream>>>(ca);
    const unsigned pblocks = blocks_for(ctx, bound, 128, 16);
    edge_visit<<<blocks_for(ctx, bound, 64, 8), 256, 0, ctx->stream>>>(ca);
    edge_own<<<pblocks, 128, 0, ctx->stream>>>(ca);
    scan_block_sums<<<1, 1024, 0, ctx->stream>>>(ca.sums, cblocks, &oa.c->mesh);
    cube_offsets<<<cblocks, 256, 0, ctx->stream>>>(ca);
    ctx->launches += 8;
    if ((s = check_launch(ctx, "dual cubes")) != ISO_OK) return s;
    LhmcTrace t{};
    while (true) {
        ca.out_v = (float*)ctx->mesh_v.p;
        ca.out_i = (uint32_t*)ctx->mesh_i.p;
        ca.out_k = keys ? (uint64_t*)ctx->mesh_k.p : nullptr;
        auto room = [](size_t n) { return (uint32_t)std::min<size_t>(n, 0xFFFFFFFFu); };
        ca.cap_v = room(keys ? std::min(ctx->mesh_v.bytes / 12, ctx->mesh_k.bytes / 16) : ctx->mesh_v.bytes / 12);
        ca.cap_t = room(ctx->mesh_i.bytes / 12);
        cube_emit<<<pblocks, 128, 0, ctx->stream>>>(ca);
        ctx->launches++;
        if ((s = check_launch(ctx, "cube_emit")) != ISO_OK) return s;
        if (rec) return ISO_OK;
        e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "read counts");
        if ((uint32_t)ctx->h_pinned[3] && (s = read_device_errors(ctx)) != ISO_OK) return s;
        t = counts_of(ctx);
        ctx->lhmc_stale = h->stale;
        if (t.nv <= ca.cap_v && t.nt <= ca.cap_t) break;
        // it did not all fit (the counts are exact): again into buffers of that size
        if ((s = ensure(ctx, ctx->mesh_v, 12ull * t.nv)) != ISO_OK) return s;
        if ((s = ensure(ctx, ctx->mesh_i, 12ull * t.nt)) != ISO_OK) return s;
        if (keys && (s = ensure(ctx, ctx->mesh_k, 16ull * t.nv)) != ISO_OK) return s;
    }
    if (trace) *trace = t;
    ctx->last.num_vertices = t.nv;
    ctx->last.num_triangles = t.nt;
    ctx->last.num_cells = t.ncubes;
    if (info) *info = ctx->last;
    return ISO_OK;
}

extern "C" uint64_t iso_lhmc_stale_corners(const iso_ctx* ctx) { return ctx ? ctx->lhmc_stale : 0; }

static void lhmc_buffers(const iso_ctx* ctx, void** b) {
    const DevBuf* bufs[6] = {&ctx->aux, &ctx->aux2, &ctx->aux3, &ctx->mesh_v, &ctx->mesh_i, &ctx->mesh_k};
    for (int i = 0; i < 6; ++i) b[i] = bufs[i]->p;
}

void iso::lhmc_plan_release(iso_ctx* ctx) {
    if (ctx->lhmc_plan.exec) cudaGraphExecDestroy(ctx->lhmc_plan.exec);
    ctx->lhmc_plan = iso_ctx::LhmcPlan{};
}

// LinearHashedMarchingCubes of a program, replaying a recorded CUDA graph when
// the same (program, depth, flags) repeats: the eager run's counts are baked
// into the recording (no synchronisation between generations), and every
// count the replay computes is checked against them before its mesh is
// used; any difference (or an error flag) falls back to the eager path.
static iso_status lhmc_planned(iso_ctx* ctx, const iso_program* prog, uint32_t depth, uint32_t flags,
                               iso_mesh_info* info) {
    if (!ctx || !prog) return ISO_ERR_INVALID_ARG;
    iso_ctx::LhmcPlan& P = ctx->lhmc_plan;
    void* bufs[6];
    lhmc_buffers(ctx, bufs);
    if (P.exec && !ctx->timing && !debug_waits_run_out() && P.prog == prog && P.prog_uid == prog->uid && P.depth == depth && P.flags == flags &&
        std::memcmp(P.bufs, bufs, sizeof(bufs)) == 0 && set_device(ctx) == ISO_OK) {
        cudaError_t e = cudaGraphLaunch(P.exec, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "octree graph");
        const LhmcTrace t = counts_of(ctx);
        const bool same = t.nodes == P.nodes && t.ncubes == P.ncubes && t.nt == P.nt && t.nv == P.nv &&
                          (uint32_t)ctx->h_pinned[3] == 0;
        if (same) {
            ctx->launches += P.launches;
            ctx->last = iso_mesh_info{P.nv, P.nt, P.ncubes};
            ctx->last_flags = flags;
            ctx->last_vertex_floats = 3;
            ctx->lhmc_stale = ((const Ctl*)(ctx->h_pinned + LHMC_PIN_CTL))->stale;
            if (info) *info = ctx->last;
            return ISO_OK;
        }
        if ((uint32_t)ctx->h_pinned[3]) cudaMemsetAsync(ctx->d_err, 0, 4, ctx->stream);
        lhmc_plan_release(ctx);
    }
    LhmcTrace tr;
    iso_status s = lhmc_extract_impl(ctx, prog, depth, flags, info, &tr, nullptr);
    if (s != ISO_OK) return s;
    const uint64_t key[3] = {prog->uid, depth, flags};
    const bool repeat = std::memcmp(key, ctx->lhmc_last_key, sizeof(key)) == 0;
    std::memcpy(ctx->lhmc_last_key, key, sizeof(key));
    if (ctx->timing || debug_waits_run_out() || !repeat) return ISO_OK;
    // record the same extraction with the counts just found
    lhmc_plan_release(ctx);
    const uint64_t launches0 = ctx->launches;
    const iso_mesh_info keep = ctx->last;
    const uint64_t keep_stale = ctx->lhmc_stale;
    if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return ISO_OK;
    }
    ctx->capturing = true;
    iso_status rs = lhmc_extract_impl(ctx, prog, depth, flags, nullptr, nullptr, &tr);
    ctx->capturing = false;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    const uint64_t recorded = ctx->launches - launches0;
    ctx->launches = launches0;
    ctx->last = keep;
    ctx->lhmc_stale = keep_stale;
    if (rs == ISO_OK && e == cudaSuccess && g) {
        cudaGraphExec_t exec = nullptr;
        if (cudaGraphInstantiate(&exec, g, 0) == cudaSuccess) {
            P.exec = exec;
            P.prog = prog;
            P.prog_uid = prog->uid;
            P.depth = depth;
            P.flags = flags;
            lhmc_buffers(ctx, P.bufs);
            P.nodes = tr.nodes;
            P.ncubes = tr.ncubes;
            P.nt = tr.nt;
            P.nv = tr.nv;
            P.launches = recorded;
        }
    }
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    ctx->last_error.clear();
    return ISO_OK;
}

// ISO_FLAG_NORMALS: the *InterleavedNormals sinks, sample_normal at every vertex
extern "C" iso_status iso_lhmc_extract(iso_ctx* ctx, const iso_program* prog, uint32_t max_depth, uint32_t flags, iso_mesh_info* info) {
    iso::NvtxRange nvtx_range("iso_lhmc_extract");
    if (!ctx || !prog) return ISO_ERR_INVALID_ARG;
    if (flags & ~(uint32_t)(ISO_FLAG_KEYS | ISO_FLAG_NORMALS)) return fail(ctx, ISO_ERR_INVALID_ARG, "unsupported flags");
    iso_status s = lhmc_planned(ctx, prog, max_depth, flags & ~(uint32_t)ISO_FLAG_NORMALS, info);
    if (s != ISO_OK || !(flags & ISO_FLAG_NORMALS)) return s;
    return attach_normals(ctx, prog);
}
