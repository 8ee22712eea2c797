// Device build of the acceleration structures, for scenes that are large or
// already on the GPU.  Takes the place of the host builder (bvh.cpp; the
// reference's driver BLAS build, WaveFrontPathTracer.cpp:202-457):
//   1. the scene box, the centroid box and the largest absolute coordinate
//      (for the conservative box growth) in one pass;
//   2. 63-bit Morton keys of the triangle centroids, sorted with the
//      library's radix sort;
//   3. PLOC (Meister and Bittner, "Parallel Locally-Ordered Clustering for
//      Bounding Volume Hierarchy Construction", IEEE TVCG 2018): every
//      cluster picks the neighbour among the 8 (knob) on either side (in
//      Morton order) whose merged box has the least surface area, mutual pairs
//      merge, the cluster list is compacted by a prefix sum, until one
//      cluster is left.  The passes run in one cooperative launch, and the
//      thread that merges a pair also writes the BVH2 node in the traversal
//      format (children's boxes grown by 2^-22 P as in the host builder;
//      single-triangle leaves) and the node's tables of the SAH collapse,
//      whose dynamic programme is bottom-up like the clustering;
//   4. the BVH8 by the host's SAH collapse, emitted top-down one level at a
//      time in a second cooperative launch, eight lanes per node, with
//      look-back allocation, so the layout is deterministic.
// The host reads the device back once, at the end (a mesh of more than
// kPassesPerLaunch clustering passes: once per launch).  Every device wait is
// bounded (kSpinLimit polls, then the timeout status); kernels check their
// indices against the buffers they write.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "build.cuh"
#include "common.cuh"
#include "scene.h"
#include "stages.cuh"

namespace wfpt {

cudaError_t status_build(uint32_t* out) { return read_and_clear_status(out); }

// PLOC search radius (clusters on either side in Morton order).  On the
// courtyard's bounce-1 rays 8 gave the fastest traversal of radii 8-64 (the
// BVH8 from radius 8 traced closest hits 8 % faster than from 16, 13 %
// faster than from 64).
static int g_ploc_radius = 8;
void set_ploc_radius(int r) { g_ploc_radius = r < 1 ? 1 : (r > 64 ? 64 : r); }
int get_ploc_radius() { return g_ploc_radius; }

namespace {

constexpr int kBB = 256;      // threads per build block
constexpr int kPlocRMax = 64;  // largest PLOC search radius (knob build.ploc.radius)
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kSlowPass = 32;  // see k_ploc
// Passes of one launch of k_ploc.  Meshes take some 20 to 100 in all; one that
// merges a pair or two per pass (a strip whose triangles get steadily smaller:
// passes grow with its length) goes on in further launches, so that no single
// one runs for long.
constexpr uint32_t kPassesPerLaunch = 256;

struct BuildStats {
    uint32_t bmin[3], bmax[3];  // order-preserving bits of the vertex box
    uint32_t cmin[3], cmax[3];  // ... of the centroid box
    uint32_t pmax;              // bits of the largest |coordinate|
    uint32_t bad_index;
    // Clustering: clusters and nodes after the last finished pass, passes, ties
    // by pairs from now on, no pair merged (cannot happen), blocks that
    // reached the pass barriers of the launch.
    uint32_t clusters, next_id, iterations, pair_ties, stuck, ploc_barrier;
    // Emission: BVH8 nodes and triangles emitted; by level parity, the tasks
    // of the next level and the triangles so far; blocks that reached the
    // level barriers; the tree is too deep.
    uint32_t nodes8, tris8, tasks[2], tris[2], emit_barrier, too_deep;
};

__device__ __forceinline__ uint32_t ord(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unord(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__device__ __forceinline__ float box_area(float4 lo, float4 hi) {
    float dx = __fsub_rn(hi.x, lo.x), dy = __fsub_rn(hi.y, lo.y), dz = __fsub_rn(hi.z, lo.z);
    return __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx)));
}

// ---------------------------------------------------------------- stage 1
// Box of triangle g; false when one of its indices is out of range (read as
// vertex 0, so that the keys and the sort can follow without a read-back;
// clustering and emission then return at once).
__device__ __forceinline__ bool tri_box(const float* __restrict__ pos, uint32_t nv, const uint32_t* __restrict__ idx,
                                        uint32_t g, float lo[3], float hi[3]) {
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        uint32_t v = idx[3 * (size_t)g + j];
        if (v >= nv) {
            ok = false;
            v = 0;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float p = pos[3 * (size_t)v + k];
            lo[k] = j == 0 ? p : fminf(lo[k], p);
            hi[k] = j == 0 ? p : fmaxf(hi[k], p);
        }
    }
    return ok;
}

__global__ void __launch_bounds__(kBB) k_tri_bounds(const float* __restrict__ pos, uint32_t nv,
                                                    const uint32_t* __restrict__ idx, uint32_t nt,
                                                    BuildStats* __restrict__ st) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t bl[3] = {kNone, kNone, kNone}, bh[3] = {0, 0, 0};
    uint32_t cl[3] = {kNone, kNone, kNone}, ch[3] = {0, 0, 0};
    uint32_t pm = 0;
    if (g < nt) {
        float lo[3], hi[3];
        if (!tri_box(pos, nv, idx, g, lo, hi)) atomicOr(&st->bad_index, 1u);
        float pmf = 0.0f;
        for (int k = 0; k < 3; ++k) {
            bl[k] = ord(lo[k]);
            bh[k] = ord(hi[k]);
            float c = __fmul_rn(0.5f, __fadd_rn(lo[k], hi[k]));
            cl[k] = ch[k] = ord(c);
            pmf = fmaxf(pmf, fmaxf(fabsf(lo[k]), fabsf(hi[k])));
        }
        pm = __float_as_uint(pmf);
    }
    for (int k = 0; k < 3; ++k) {
        bl[k] = __reduce_min_sync(0xffffffffu, bl[k]);
        bh[k] = __reduce_max_sync(0xffffffffu, bh[k]);
        cl[k] = __reduce_min_sync(0xffffffffu, cl[k]);
        ch[k] = __reduce_max_sync(0xffffffffu, ch[k]);
    }
    pm = __reduce_max_sync(0xffffffffu, pm);
    // Block reduction of the 13 values (one atomic per value and block:
    // per-warp atomics on the same 13 words serialised on 3M triangles).
    __shared__ uint32_t s_red[kBB / 32][13];
    const uint32_t warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        for (int k = 0; k < 3; ++k) {
            s_red[warp][k] = bl[k];
            s_red[warp][3 + k] = bh[k];
            s_red[warp][6 + k] = cl[k];
            s_red[warp][9 + k] = ch[k];
        }
        s_red[warp][12] = pm;
    }
    __syncthreads();
    if (threadIdx.x < 13) {
        const uint32_t q = threadIdx.x;
        const bool is_min = q < 3 || (q >= 6 && q < 9);
        uint32_t v = s_red[0][q];
        for (int w = 1; w < kBB / 32; ++w) v = is_min ? min(v, s_red[w][q]) : max(v, s_red[w][q]);
        uint32_t* dst = q < 3 ? &st->bmin[q] : q < 6 ? &st->bmax[q - 3] : q < 9 ? &st->cmin[q - 6]
                      : q < 12 ? &st->cmax[q - 9] : &st->pmax;
        if (is_min) atomicMin(dst, v);
        else atomicMax(dst, v);
    }
}

// ---------------------------------------------------------------- stage 2
__device__ __forceinline__ uint64_t spread21(uint32_t x) {
    uint64_t v = x & 0x1FFFFFu;
    v = (v | (v << 32)) & 0x1F00000000FFFFull;
    v = (v | (v << 16)) & 0x1F0000FF0000FFull;
    v = (v | (v << 8)) & 0x100F00F00F00F00Full;
    v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

__global__ void __launch_bounds__(kBB) k_centroid_keys(const float* __restrict__ pos, uint32_t nv,
                                                       const uint32_t* __restrict__ idx, uint32_t nt,
                                                       const BuildStats* __restrict__ st, uint64_t* __restrict__ keys,
                                                       uint32_t* __restrict__ vals) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nt) return;
    float lo[3], hi[3];
    tri_box(pos, nv, idx, g, lo, hi);
    uint32_t q[3];
    for (int k = 0; k < 3; ++k) {
        const float c = __fmul_rn(0.5f, __fadd_rn(lo[k], hi[k]));
        const float a = unord(st->cmin[k]), b = unord(st->cmax[k]);
        const float ext = __fsub_rn(b, a);
        float t = ext > 0.0f ? __fdiv_rn(__fsub_rn(c, a), ext) : 0.0f;
        t = fminf(fmaxf(t, 0.0f), 1.0f);
        q[k] = min((uint32_t)__fmul_rn(t, 2097151.0f), 2097151u);
    }
    keys[g] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
    vals[g] = g;
}

// Leaves in Morton order: node i is the triangle vals[i]; its record goes to
// slot i of the BVH2 triangle table, its box to boxes[2 i], boxes[2 i + 1].
__global__ void __launch_bounds__(kBB) k_leaves(const uint32_t* __restrict__ vals, uint32_t nt,
                                                const float* __restrict__ pos, uint32_t nv,
                                                const uint32_t* __restrict__ idx,
                                                const uint32_t* __restrict__ geom_first, uint32_t ngeom,
                                                float4* __restrict__ boxes, float4* __restrict__ recs,
                                                uint32_t* __restrict__ clusters) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt) return;
    const uint32_t g = vals[i];
    if (g >= nt) {
        raise_status(kErrBounds);
        return;
    }
    // Geometry: the last entry of geom_first that is <= g (upper_bound - 1).
    uint32_t a = 0, b = ngeom;
    while (a < b) {
        uint32_t mid = (a + b) >> 1;
        if (geom_first[mid] <= g) a = mid + 1;
        else b = mid;
    }
    const uint32_t geom = a == 0 ? 0 : a - 1;
    const uint32_t prim = g - geom_first[geom];
    float4 r[3];
    for (int j = 0; j < 3; ++j) {
        uint32_t v = idx[3 * (size_t)g + j];
        if (v >= nv) v = 0;
        r[j] = make_float4(pos[3 * (size_t)v], pos[3 * (size_t)v + 1], pos[3 * (size_t)v + 2], 0.0f);
    }
    boxes[2 * (size_t)i] = make_float4(fminf(fminf(r[0].x, r[1].x), r[2].x), fminf(fminf(r[0].y, r[1].y), r[2].y),
                                       fminf(fminf(r[0].z, r[1].z), r[2].z), 0.0f);
    boxes[2 * (size_t)i + 1] = make_float4(fmaxf(fmaxf(r[0].x, r[1].x), r[2].x), fmaxf(fmaxf(r[0].y, r[1].y), r[2].y),
                                           fmaxf(fmaxf(r[0].z, r[1].z), r[2].z), 0.0f);
    r[0].w = __int_as_float((int32_t)prim);
    r[1].w = __int_as_float((int32_t)geom);
    r[2].w = __uint_as_float(g);
    recs[3 * (size_t)i + 0] = r[0];
    recs[3 * (size_t)i + 1] = r[1];
    recs[3 * (size_t)i + 2] = r[2];
    clusters[i] = i;
}

// ----------------------------------------------- waits between the blocks
// of a cooperative launch (all of them resident at once).

// Exclusive prefix over the tiles before `tile` of two counts packed as
// hi << 28 | lo (totals below 2^27 and 2^28) by decoupled look-back, 32
// predecessors per round trip; called by one full warp, result in all lanes.
// A state holds epoch (7 bits, the pass or level: states are not cleared in
// between) | flag (1 aggregate, 2 inclusive prefix) | hi | lo.
constexpr int kStFlag = 55, kStEpoch = 57;
constexpr uint64_t kStValue = (1ull << kStFlag) - 1;
__device__ __forceinline__ uint64_t pack_state(uint32_t epoch, uint64_t flag, uint64_t v) {
    return ((uint64_t)(epoch & 127u) << kStEpoch) | (flag << kStFlag) | v;
}
__device__ uint64_t tile_prefix64(unsigned long long* state, uint32_t tile, uint64_t v, uint32_t epoch) {
    const uint32_t lane = threadIdx.x & 31;
    if (lane == 0) atomicExch(&state[tile], (unsigned long long)pack_state(epoch, tile == 0 ? 2 : 1, v));
    if (tile == 0) return 0;
    uint64_t excl = 0;
    uint32_t spins = 0;
    int32_t top = (int32_t)tile - 1;
    for (;;) {
        const int32_t t = top - (int32_t)lane;
        uint64_t s = pack_state(epoch, 2, 0);  // before tile 0: a prefix of 0
        if (t >= 0) s = *((volatile unsigned long long*)&state[t]);
        const uint32_t flag =
            (uint32_t)(s >> kStEpoch) == (epoch & 127u) ? (uint32_t)(s >> kStFlag) & 3u : 0u;
        const uint32_t pref = __ballot_sync(0xffffffffu, flag == 2u);
        const uint32_t unset = __ballot_sync(0xffffffffu, flag == 0u);
        const uint32_t p = pref ? (uint32_t)__ffs(pref) - 1u : 32u;
        const uint32_t upto = p < 31u ? ((2u << p) - 1u) : 0xffffffffu;  // lanes 0..p
        if (unset & upto) {
            if (++spins > kSpinLimit) {
                raise_status(kErrTimeout);
                break;
            }
            continue;
        }
        const uint64_t w = lane <= p ? (s & kStValue) : 0u;
        excl += ((uint64_t)__reduce_add_sync(0xffffffffu, (uint32_t)(w >> 28)) << 28) +
                __reduce_add_sync(0xffffffffu, (uint32_t)w & 0xFFFFFFFu);
        if (p < 32u) break;
        top -= 32;
    }
    if (lane == 0) atomicExch(&state[tile], (unsigned long long)pack_state(epoch, 2, (excl + v) & kStValue));
    return excl;
}

// All `blocks` blocks arrive (the counter reaches `target`, the sum of the
// arrivals of all barriers so far); what they wrote before is visible after.
// False after a timeout.
__device__ bool block_barrier(uint32_t* counter, uint32_t target) {
    __shared__ uint32_t s_ok;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(counter, 1u);
        uint32_t ok = 1, spins = 0;
        while ((int32_t)(*((volatile uint32_t*)counter) - target) < 0) {
            if (++spins > kSpinLimit) {
                raise_status(kErrTimeout);
                ok = 0;
                break;
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Exclusive scan of one word per thread over the block (two 16-bit counts
// that do not overflow into each other); *total receives the block's sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t off = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < kBB / 32; ++w) {
        const uint32_t c = s_warp[w];
        if (w < (int)warp) off += c;
        sum += c;
    }
    *total = sum;
    return off + x - v;
}

// ---------------------------------------------------------------- stage 3
// Collapse tables of a BVH2 node (the host's plan_sah): cost[2 i], [2 i + 1]
// are the least costs of node i's subtree with at most 1..8 BVH8 children;
// meta[i] = {how[0..3], how[4..7], triangles, split8}: byte how[0] is -1 for
// one leaf child, 0 for one inner child; how[s-1] (s > 1) 0 for the same as
// s-1, a > 0 for a slots to child 0; split8 is child 0's slots when the node
// is a BVH8 inner node.
struct Grown {
    float4 lo, hi;
};

// BVH2 node `index` over clusters a and b (ids: below n a triangle, above an
// inner node stored at index 2 n - 2 - id, so that the root, merged last, is
// node 0 and children come after their parents), and its collapse tables.
__device__ __forceinline__ void write_node2(uint32_t index, uint32_t n, const uint32_t id[2], const float4 lo[2],
                                            const float4 hi[2], float delta, bool want8, float tri_cost,
                                            float4* __restrict__ nodes2, float4* cost, uint4* meta) {
    const uint32_t last = 2 * n - 2;
    Grown g[2];
    int32_t link[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        g[c].lo = make_float4(__fsub_rn(lo[c].x, delta), __fsub_rn(lo[c].y, delta), __fsub_rn(lo[c].z, delta), 0.0f);
        g[c].hi = make_float4(__fadd_rn(hi[c].x, delta), __fadd_rn(hi[c].y, delta), __fadd_rn(hi[c].z, delta), 0.0f);
        link[c] = id[c] < n ? (int32_t)~(id[c] << 3) : (int32_t)(last - id[c]);
    }
    float4* o = nodes2 + 4 * (size_t)index;
    o[0] = make_float4(g[0].lo.x, g[0].hi.x, g[0].lo.y, g[0].hi.y);
    o[1] = make_float4(g[1].lo.x, g[1].hi.x, g[1].lo.y, g[1].hi.y);
    o[2] = make_float4(g[0].lo.z, g[0].hi.z, g[1].lo.z, g[1].hi.z);
    o[3] = make_float4(__int_as_float(link[0]), __int_as_float(link[1]), 0.0f, 0.0f);
    if (!want8) return;
    float cc[2][8];
    uint32_t tris = 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (link[c] < 0) {
            const float a = __fmul_rn(box_area(g[c].lo, g[c].hi), tri_cost);
#pragma unroll
            for (int s = 0; s < 8; ++s) cc[c][s] = a;
            tris += 1;
        } else {
            const float4 x = __ldcg(&cost[2 * (size_t)link[c]]), y = __ldcg(&cost[2 * (size_t)link[c] + 1]);
            cc[c][0] = x.x; cc[c][1] = x.y; cc[c][2] = x.z; cc[c][3] = x.w;
            cc[c][4] = y.x; cc[c][5] = y.y; cc[c][6] = y.z; cc[c][7] = y.w;
            tris += __ldcg(&meta[link[c]]).z;
        }
    }
    const float4 ulo = make_float4(fminf(g[0].lo.x, g[1].lo.x), fminf(g[0].lo.y, g[1].lo.y), fminf(g[0].lo.z, g[1].lo.z), 0.0f);
    const float4 uhi = make_float4(fmaxf(g[0].hi.x, g[1].hi.x), fmaxf(g[0].hi.y, g[1].hi.y), fmaxf(g[0].hi.z, g[1].hi.z), 0.0f);
    const float A = box_area(ulo, uhi);
    const float inf = __int_as_float(0x7f800000);
    float dist[9];
    uint32_t arg[9];
#pragma unroll
    for (int j = 2; j <= 8; ++j) {
        dist[j] = inf;
        arg[j] = 1;
#pragma unroll
        for (int a = 1; a < j; ++a) {
            const float c = __fadd_rn(cc[0][a - 1], cc[1][j - a - 1]);
            if (c < dist[j]) {
                dist[j] = c;
                arg[j] = a;
            }
        }
    }
    const float c_inner = __fadd_rn(A, dist[8]);
    const float c_leaf = tris <= 3 ? __fmul_rn(__fmul_rn(A, (float)tris), tri_cost) : inf;
    float out[8];
    uint32_t how[2] = {c_leaf <= c_inner ? 0xFFu : 0u, 0u};
    out[0] = fminf(c_leaf, c_inner);
#pragma unroll
    for (int s = 2; s <= 8; ++s) {
        const bool split = dist[s] < out[s - 2];
        out[s - 1] = split ? dist[s] : out[s - 2];
        how[(s - 1) >> 2] |= (split ? arg[s] : 0u) << (8 * ((s - 1) & 3));
    }
    __stcg(&cost[2 * (size_t)index], make_float4(out[0], out[1], out[2], out[3]));
    __stcg(&cost[2 * (size_t)index + 1], make_float4(out[4], out[5], out[6], out[7]));
    __stcg(&meta[index], make_uint4(how[0], how[1], tris, arg[8]));
}

__device__ __forceinline__ bool same_box(const float4* s_lo, const float4* s_hi, int a, int b) {
    const float4 alo = s_lo[a], ahi = s_hi[a], blo = s_lo[b], bhi = s_hi[b];
    return alo.x == blo.x && alo.y == blo.y && alo.z == blo.z && ahi.x == bhi.x && ahi.y == bhi.y && ahi.z == bhi.z;
}

// The position of the R on either side of position i (box `at` in shared
// memory) whose box merged with i's has the least surface area.  Ties go to the
// positions of i's own run of equal boxes first, and among these to the one with
// the least i xor j: so coincident triangles, which follow one another in Morton
// order, pair up as (2 k, 2 k + 1).  Other ties go to the smaller position, or
// (PAIR_TIES) also to the least i xor j.
template <bool PAIR_TIES>
__device__ __forceinline__ uint32_t nearest(const float4* s_lo, const float4* s_hi, int at, int R, int i, uint32_t m) {
    const float4 alo = s_lo[at], ahi = s_hi[at];
    uint32_t best = kNone, nn = kNone;
    const int d0 = max(-R, -i), d1 = min(R, (int)m - 1 - i);
    for (int d = d0; d <= d1; ++d) {
        if (d == 0) continue;
        const float4 blo = s_lo[at + d], bhi = s_hi[at + d];
        const float4 ulo = make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), 0.0f);
        const float4 uhi = make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.0f);
        const uint32_t key = __float_as_uint(box_area(ulo, uhi)), j = (uint32_t)(i + d);
        if (key < best || (PAIR_TIES && key == best && ((uint32_t)i ^ j) < ((uint32_t)i ^ nn))) {
            best = key;
            nn = j;
        }
    }
    // Only where the merged box is no larger than this one may it be an equal one's.
    if (best == __float_as_uint(box_area(alo, ahi))) {
        uint32_t tie = kNone;
        for (int side = -1; side <= 1; side += 2)
            for (int d = side; d0 <= d && d <= d1 && same_box(s_lo, s_hi, at, at + d); d += side) {
                const uint32_t j = (uint32_t)(i + d), x = (uint32_t)i ^ j;
                if (x < tie) {
                    tie = x;
                    nn = j;
                }
            }
    }
    return nn;
}

// Where a launch of k_ploc goes on (as in BuildStats).
struct PlocStart {
    uint32_t clusters, next_id, iterations, pair_ties;
};

// The whole clustering.  A block takes tiles of kBB - 2 R cluster positions
// and holds the boxes of the tile and of 2 R positions on either side in
// shared memory: enough to find the nearest neighbour (see nearest) of every
// position of the tile and of the R on either side, hence the mutual pairs that
// start or end in the tile.  For a fixed cluster that order is an order of pairs
// (area; runs of equal boxes first; i xor j or the positions), so the pair that
// is least in it over all pairs is mutual and every pass merges at least one.
// No more than one, where all ties go to the smaller position: 600 coincident
// triangles took 599 passes and gave a chain too deep for the emission and for
// the traversal's stacks, and 80 of them in the courtyard's mesh a tree of depth
// 100.  Runs of equal boxes first: 10 passes, and depth 29.  A strip of 40,000 equal
// triangles still took over 20,000 passes; so after a pass that merged less
// than one in kSlowPass of its clusters the other ties go by i xor j too: 22
// passes.  Triangle soups, the courtyard and the city merge 9 % and more at
// every radius, a regular grid 6 % at radius 8: their trees are those of the
// smaller position.
// A pair's node is made by the block of its lower position, the first
// threads of the block taking one pair each.  The pass ends at a barrier of
// the blocks that had a tile; blocks without one are done for good, since
// the list only shrinks, and once one tile is left its block goes on alone.
//
// Bound by latency: 3M triangles take 53 passes, the 40 last of them with
// less than one tile per SM, each a chain of a few dependent L2 round trips
// (28 % issue active, 1.1 TB/s).  0.79 ms, against 0.97 ms for the same passes
// as separate kernels (neighbours, flags, a three-launch prefix sum, merge)
// with as much again in launches and a host read-back per pass, plus 0.82 ms
// for the BVH2 nodes and the collapse tables in kernels of their own.  Four
// blocks per SM: whole 3M build 2.68 ms with three, 2.58 with four, 2.59 with
// five.
__global__ void __launch_bounds__(kBB, 4) k_ploc(uint32_t* cl_a, uint32_t* cl_b, uint32_t n, int radius,
                                                 float4* boxes, float4* __restrict__ nodes2, float4* cost,
                                                 uint4* meta, int want8, float tri_cost, unsigned long long* state,
                                                 BuildStats* st, PlocStart from) {
    constexpr int kMost = kBB + 2 * kPlocRMax;
    __shared__ float4 s_lo[kMost], s_hi[kMost];
    __shared__ uint32_t s_id[kMost], s_nn[kBB], s_pair[kBB], s_warp[kBB / 32];
    __shared__ unsigned long long s_base;
    const int R = radius < 1 ? 1 : (radius > kPlocRMax ? kPlocRMax : radius);
    const int T = kBB - 2 * R;
    const int tid = (int)threadIdx.x;
    const uint32_t cap = 2 * n - 1;
    const float delta = __fmul_rn(__uint_as_float(st->pmax), 0x1p-22f);
    uint32_t m = from.clusters, next_id = from.next_id, iter = from.iterations, target = 0;
    bool pair_ties = from.pair_ties != 0;
    if (st->bad_index) return;  // refused by the host: the triangles may all be one
    while (m > 1) {
        const uint32_t ntiles = (m + T - 1) / T;
        const uint32_t nblocks = min(gridDim.x, ntiles);
        if (blockIdx.x >= nblocks) return;
        const uint32_t* cin = (iter & 1) ? cl_b : cl_a;
        uint32_t* cout = (iter & 1) ? cl_a : cl_b;
        for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const int b0 = (int)tile * T;
            for (int t = tid; t < kBB + 2 * R; t += kBB) {
                const int j = b0 - 2 * R + t;
                if (j >= 0 && j < (int)m) {
                    const uint32_t id = __ldcg(&cin[j]);
                    s_id[t] = id;
                    if (id < cap) {
                        s_lo[t] = __ldcg(&boxes[2 * (size_t)id]);
                        s_hi[t] = __ldcg(&boxes[2 * (size_t)id + 1]);
                    }
                }
            }
            __syncthreads();
            const int i = b0 - R + tid;
            uint32_t nn = kNone;
            if (i >= 0 && i < (int)m) nn = pair_ties ? nearest<true>(s_lo, s_hi, tid + R, R, i, m) : nearest<false>(s_lo, s_hi, tid + R, R, i, m);
            s_nn[tid] = nn;
            __syncthreads();
            bool keep = false, merge = false;
            if (tid >= R && tid < R + T && i < (int)m) {
                const bool mutual = nn != kNone && s_nn[tid + ((int)nn - i)] == (uint32_t)i;
                merge = mutual && i < (int)nn;
                keep = !(mutual && i > (int)nn);
            }
            uint32_t total;
            const uint32_t rank = block_scan(((uint32_t)merge << 16) | (uint32_t)keep, s_warp, &total);
            const uint32_t pairs = total >> 16, kept = total & 0xFFFFu;
            if (tid < 32) {
                const uint64_t p = tile_prefix64(state, tile, ((uint64_t)pairs << 28) | kept, iter);
                if (tid == 0) s_base = p;
            }
            if (merge) s_pair[rank >> 16] = (uint32_t)tid;
            __syncthreads();
            const uint32_t id0 = next_id + (uint32_t)(s_base >> 28), pos0 = (uint32_t)s_base & 0xFFFFFFFu;
            if (keep) {
                const uint32_t at = pos0 + (rank & 0xFFFFu);
                if (at < m) __stcg(&cout[at], merge ? id0 + (rank >> 16) : s_id[tid + R]);
                else raise_status(kErrBounds);
            }
            if (tid < (int)pairs) {
                const int t = (int)s_pair[tid], li = t + R, lj = li + ((int)s_nn[t] - (b0 - R + t));
                const uint32_t id = id0 + (uint32_t)tid;
                const uint32_t kid[2] = {s_id[li], s_id[lj]};
                if (id < cap && kid[0] < id && kid[1] < id) {
                    const float4 lo[2] = {s_lo[li], s_lo[lj]}, hi[2] = {s_hi[li], s_hi[lj]};
                    __stcg(&boxes[2 * (size_t)id], make_float4(fminf(lo[0].x, lo[1].x), fminf(lo[0].y, lo[1].y), fminf(lo[0].z, lo[1].z), 0.0f));
                    __stcg(&boxes[2 * (size_t)id + 1], make_float4(fmaxf(hi[0].x, hi[1].x), fmaxf(hi[0].y, hi[1].y), fmaxf(hi[0].z, hi[1].z), 0.0f));
                    write_node2(2 * n - 2 - id, n, kid, lo, hi, delta, want8 != 0, tri_cost, nodes2, cost, meta);
                } else {
                    raise_status(kErrBounds);
                }
            }
            if (tile == ntiles - 1 && tid == 0) {
                st->clusters = pos0 + kept;
                st->next_id = id0 + pairs;
            }
            __syncthreads();
        }
        target += nblocks;
        if (nblocks > 1 && !block_barrier(&st->ploc_barrier, target)) return;
        const uint32_t left = __ldcg(&st->clusters);
        next_id = __ldcg(&st->next_id);
        ++iter;
        pair_ties = pair_ties || m - left < m / kSlowPass;
        if (blockIdx.x == 0 && tid == 0) {
            st->iterations = iter;
            st->pair_ties = pair_ties;
            if (left >= m) st->stuck = 1;
        }
        if (left >= m || iter - from.iterations == kPassesPerLaunch) return;
        m = left;
        // A lone block rewrites st->clusters in its next pass: not before
        // every thread has read it.
        __syncthreads();
    }
}

// ---------------------------------------------------------------- stage 4
// Triangles of a leaf child (a subtree of at most three triangles), depth
// first, child 0 first, like the host's gather_tris.
__device__ int gather3(const Bvh2Node* __restrict__ nodes, int32_t link, uint32_t* recs) {
    int32_t st[8];
    int sp = 0, cnt = 0;
    st[sp++] = link;
    while (sp > 0) {
        const int32_t l = st[--sp];
        if (l < 0) {
            const uint32_t code = ~(uint32_t)l;
            const uint32_t first = code >> 3, c = (code & 7u) + 1u;
            for (uint32_t q = 0; q < c && cnt < 3; ++q) recs[cnt++] = first + q;
            continue;
        }
        const int2 kids = *reinterpret_cast<const int2*>(nodes[l].link);
        if (sp + 2 > 8) break;
        st[sp++] = kids.y;
        st[sp++] = kids.x;
    }
    return cnt;
}

__device__ __forceinline__ uint32_t how_of(const uint4& m, int s) {  // byte how[s - 1]
    return ((s <= 4 ? m.x : m.y) >> (8 * ((s - 1) & 3))) & 0xFFu;
}

// The whole emission, a level of BVH8 nodes per round: eight lanes per node,
// 32 nodes per block and tile.
//  - Children: a node's eight slots are the lanes of its group.  Each lane
//    walks from the node to the child that covers its slot, going to child 0
//    or 1 by the slots that the tables give each; lanes of one child make the
//    same steps, and the first of them owns it (so children are in lane
//    order, child 0's share first, as the host collects them).
//  - Node box, quantisation grid and the greedy slot assignment (descending
//    octant score, ties to the lower (child, slot) pair, as the host's stable
//    sort) by shuffles in the group; then lane = slot.
//  - A tile's inner children and triangles get their places by look-back over
//    the level's tiles, in task order.
// The level's children are the next level's tasks; a barrier of all blocks
// ends a level.  One thread per node, with the children collected twice (once
// to count) and a prefix sum and a read-back per level, took 1.24 ms for 3M
// triangles; this takes 0.47 ms.
constexpr int kEmitTile = kBB / 8;
// Levels below the root.  Meshes of millions of triangles have about ten;
// a few hundred triangles nested in one another are a chain, and refused.
constexpr uint32_t kMostLevels = 64;
__global__ void __launch_bounds__(kBB, 4) k_emit8(uint32_t* tasks_a, uint32_t* tasks_b, uint32_t n,
                                                  const Bvh2Node* __restrict__ nodes, const uint4* __restrict__ meta,
                                                  const float4* __restrict__ recs2, float4* __restrict__ out,
                                                  float4* __restrict__ recs8, unsigned long long* state,
                                                  BuildStats* st) {
    __shared__ uint32_t s_warp[kBB / 32];
    __shared__ unsigned long long s_base;
    __shared__ uint8_t s_at[kBB];
    __shared__ __align__(16) uint8_t s_node[kEmitTile][80];
    const uint32_t lane = threadIdx.x & 31, l = lane & 7, group = lane & 24u, slot_group = threadIdx.x >> 3;
    const uint32_t node_cap = n - 1;
    const float inf = __int_as_float(0x7f800000);
    uint32_t ntasks = 1, level_base = 0, tri_base0 = 0, target = 0;
    if (st->bad_index || st->clusters != 1) return;
    for (uint32_t level = 0; ntasks > 0; ++level) {
        if (level > kMostLevels) {
            if (blockIdx.x == 0 && threadIdx.x == 0) st->too_deep = 1;
            return;
        }
        if (ntasks > node_cap || level_base + ntasks > node_cap) {  // cannot happen
            if (blockIdx.x == 0 && threadIdx.x == 0) st->stuck = 1;
            return;
        }
        const uint32_t* tin = (level & 1) ? tasks_b : tasks_a;
        uint32_t* tout = (level & 1) ? tasks_a : tasks_b;
        const uint32_t node_base = level_base + ntasks;  // the next level's first node
        const uint32_t ntiles = (ntasks + kEmitTile - 1) / kEmitTile;
        for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
            const uint32_t task = tile * kEmitTile + slot_group;
            const bool valid = task < ntasks;
            // This lane's child.
            uint32_t p = 0, k = 0, pos = 0, ntri = 0;
            int32_t link = 0;
            bool leaf = false;
            if (valid) {
                p = level == 0 ? 0u : __ldcg(&tin[task]);
                if (p >= node_cap) {
                    raise_status(kErrBounds);
                    p = 0;
                }
                int s = (int)meta[p].w;
                if ((int)l >= s) {
                    k = 1;
                    pos = (uint32_t)s;
                    s = 8 - s;
                }
                for (int step = 0; step < 8; ++step) {
                    link = nodes[p].link[k];
                    if (link < 0) {
                        leaf = true;
                        ntri = ((~(uint32_t)link) & 7u) + 1u;
                        break;
                    }
                    const uint4 h = meta[link];
                    while (s > 1 && how_of(h, s) == 0) --s;
                    if (s <= 1) {
                        leaf = how_of(h, 1) == 0xFFu;
                        ntri = leaf ? h.z : 0u;
                        break;
                    }
                    const int a = (int)how_of(h, s);
                    p = (uint32_t)link;
                    k = (int)(l - pos) < a ? 0u : 1u;
                    if (k == 0) {
                        s = a;
                    } else {
                        s -= a;
                        pos += (uint32_t)a;
                    }
                }
            }
            const bool child = valid && l == pos;
            // Places of the tile's inner children and triangles.
            uint32_t total;
            const uint32_t mine = child ? (leaf ? ntri : 1u << 16) : 0u;
            const uint32_t before = block_scan(mine, s_warp, &total);
            if (threadIdx.x < 32) {
                const uint64_t q = tile_prefix64(state, tile, ((uint64_t)(total >> 16) << 28) | (total & 0xFFFFu), level);
                if (threadIdx.x == 0) s_base = q;
            }
            // Box of the child (empty when this lane owns none).
            float lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf};
            if (child) {
                const float4* f = reinterpret_cast<const float4*>(&nodes[p]);
                const float4 xy = f[k];
                const float2 z = reinterpret_cast<const float2*>(f + 2)[k];
                lo[0] = xy.x; hi[0] = xy.y; lo[1] = xy.z; hi[1] = xy.w; lo[2] = z.x; hi[2] = z.y;
            }
            float nlo[3], nhi[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                nlo[a] = lo[a];
                nhi[a] = hi[a];
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) {
                    nlo[a] = fminf(nlo[a], __shfl_xor_sync(0xffffffffu, nlo[a], o));
                    nhi[a] = fmaxf(nhi[a], __shfl_xor_sync(0xffffffffu, nhi[a], o));
                }
            }
            // Quantisation grid (the host's emit_children): the smallest
            // power-of-two scale whose 255 steps from the box minimum reach
            // the box maximum; lane a of the group finds axis a's.
            int ex = -126;
            {
                const float b0 = l == 0 ? nlo[0] : (l == 1 ? nlo[1] : nlo[2]);
                const float b1 = l == 0 ? nhi[0] : (l == 1 ? nhi[1] : nhi[2]);
                const float ext = __fsub_rn(b1, b0);
                if (ext > 0.0f) {
                    int e2;
                    frexpf(__fdiv_rn(ext, 255.0f), &e2);
                    ex = e2;
                }
                for (int guard = 0; guard < 300; ++guard) {
                    ex = max(-126, min(127, ex));
                    if (__fadd_rn(b0, __fmul_rn(255.0f, ldexpf(1.0f, ex))) >= b1 || ex == 127) break;
                    ++ex;
                }
            }
            int exs[3];
            float scale[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                exs[a] = __shfl_sync(0xffffffffu, ex, (int)group + a);
                scale[a] = ldexpf(1.0f, exs[a]);
            }
            // Slots.
            float off[3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
                off[a] = __fsub_rn(__fmul_rn(0.5f, __fadd_rn(lo[a], hi[a])), __fmul_rn(0.5f, __fadd_rn(nlo[a], nhi[a])));
            uint32_t open = 0xFFu, slot = 8u;
            s_at[threadIdx.x] = 0xFF;
            __syncwarp();
            for (int round = 0; round < 8; ++round) {
                const bool want = child && slot == 8u;
                if (!__any_sync(0xffffffffu, want)) break;
                float best = 0.0f;
                uint32_t bs = 8u;
#pragma unroll
                for (uint32_t sl = 0; sl < 8; ++sl) {
                    float sc = __fadd_rn(0.0f, (sl & 1u) ? -off[0] : off[0]);
                    sc = __fadd_rn(sc, (sl & 2u) ? -off[1] : off[1]);
                    sc = __fadd_rn(sc, (sl & 4u) ? -off[2] : off[2]);
                    if (((open >> sl) & 1u) && (bs == 8u || sc > best)) {
                        best = sc;
                        bs = sl;
                    }
                }
                const uint32_t key = want ? ord(__fadd_rn(best, 0.0f)) : 0u;
                uint32_t top = key;
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
                const uint32_t won = (__ballot_sync(0xffffffffu, want && key == top) >> group) & 0xFFu;
                const uint32_t first = won ? (uint32_t)__ffs(won) - 1u : 0u;
                const uint32_t taken = __shfl_sync(0xffffffffu, bs, (int)(group + first));
                if (won) {
                    open &= ~(1u << taken);
                    if (l == first) {
                        slot = bs;
                        s_at[(threadIdx.x & ~7u) + bs] = (uint8_t)l;
                    }
                }
            }
            __syncwarp();
            // From here on lane = slot.
            const uint32_t src = s_at[threadIdx.x];
            const bool has = src < 8u;
            const int from = (int)(group + (src & 7u));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                lo[a] = __shfl_sync(0xffffffffu, lo[a], from);
                hi[a] = __shfl_sync(0xffffffffu, hi[a], from);
            }
            link = __shfl_sync(0xffffffffu, link, from);
            leaf = __shfl_sync(0xffffffffu, (int)leaf, from) != 0 && has;
            ntri = __shfl_sync(0xffffffffu, ntri, from);
            if (!leaf) ntri = 0u;
            const bool inner = has && !leaf;
            uint32_t tri_off = ntri;  // inclusive scan over the slots
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, tri_off, o, 8);
                if (l >= (uint32_t)o) tri_off += y;
            }
            tri_off -= ntri;
            const uint32_t imask = (__ballot_sync(0xffffffffu, inner) >> group) & 0xFFu;
            const uint32_t inner_i = __popc(imask & ((1u << l) - 1u));
            __syncthreads();  // s_base
            const uint32_t at = __shfl_sync(0xffffffffu, before, (int)group);
            const uint32_t inner_off = (uint32_t)(s_base >> 28) + (at >> 16);
            const uint32_t tri_base = tri_base0 + ((uint32_t)s_base & 0xFFFFFFFu) + (at & 0xFFFFu);
            uint8_t* const img = s_node[slot_group];
            uint8_t mt = 0;
            if (leaf) mt = (uint8_t)(((ntri == 1 ? 1u : (ntri == 2 ? 3u : 7u)) << 5) | tri_off);
            if (inner) mt = (uint8_t)((1u << 5) | (24u + l));
            img[24 + l] = mt;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                int ql = 0, qh = 0;
                if (has) {
                    const float sc = scale[a];
                    ql = (int)fmaxf(0.0f, fminf(255.0f, floorf(__fdiv_rn(__fsub_rn(lo[a], nlo[a]), sc))));
                    qh = (int)fmaxf(0.0f, fminf(255.0f, ceilf(__fdiv_rn(__fsub_rn(hi[a], nlo[a]), sc))));
                    while (ql > 0 && __fadd_rn(nlo[a], __fmul_rn((float)ql, sc)) > lo[a]) --ql;
                    while (qh < 255 && __fadd_rn(nlo[a], __fmul_rn((float)qh, sc)) < hi[a]) ++qh;
                }
                img[32 + 8 * a + l] = (uint8_t)ql;
                img[56 + 8 * a + l] = (uint8_t)qh;
            }
            if (l == 0) {
                float* h = reinterpret_cast<float*>(img);
                h[0] = nlo[0];
                h[1] = nlo[1];
                h[2] = nlo[2];
                uint32_t* w = reinterpret_cast<uint32_t*>(img);
                w[3] = (uint32_t)(exs[0] + 127) | ((uint32_t)(exs[1] + 127) << 8) | ((uint32_t)(exs[2] + 127) << 16) | (imask << 24);
                w[4] = node_base + inner_off;
                w[5] = tri_base;
            }
            __syncwarp();
            if (valid && l < 5) out[5 * (size_t)(level_base + task) + l] = reinterpret_cast<const float4*>(img)[l];
            if (inner) {
                if (node_base + inner_off + inner_i < node_cap) __stcg(&tout[inner_off + inner_i], (uint32_t)link);
                else raise_status(kErrBounds);
            }
            if (leaf) {
                uint32_t r[3];
                const int cnt = gather3(nodes, link, r);
                for (int q = 0; q < cnt; ++q) {
                    const uint32_t dst = tri_base + tri_off + (uint32_t)q;
                    if (dst >= n || r[q] >= n) {
                        raise_status(kErrBounds);
                        continue;
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) recs8[3 * (size_t)dst + c] = recs2[3 * (size_t)r[q] + c];
                }
            }
            if (tile == ntiles - 1 && threadIdx.x == 0) {
                const uint32_t tris = tri_base0 + ((uint32_t)s_base & 0xFFFFFFFu) + (total & 0xFFFFu);
                st->tasks[level & 1] = (uint32_t)(s_base >> 28) + (total >> 16);
                st->tris[level & 1] = tris;
                st->tris8 = tris;
                st->nodes8 = node_base;
            }
            __syncthreads();
        }
        target += gridDim.x;
        if (!block_barrier(&st->emit_barrier, target)) return;
        // (By parity: a slot is written again two levels on, after every
        // block has read it and reached the next barrier.)
        level_base = node_base;
        ntasks = __ldcg(&st->tasks[level & 1]);
        tri_base0 = __ldcg(&st->tris[level & 1]);
    }
}

unsigned blocks(uint64_t n) { return (unsigned)((n + kBB - 1) / kBB); }

// Cooperative launch of as many blocks as are resident at once, at most `want`.
template <typename... Args>
cudaError_t launch_resident(void (*kernel)(Args...), uint64_t want, cudaStream_t s, Args... args) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBB, 0);
    if (e != cudaSuccess) return e;
    const uint64_t most = std::max<uint64_t>(1, (uint64_t)sms * (uint64_t)per_sm);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min(most, want));
    void* argv[] = {(void*)&args...};
    e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(kBB), argv, 0, s);
    count_launch();
    return e;
}

// Offsets into the build's one temporary allocation.
struct Arena {
    size_t bytes = 0;
    size_t take(size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) & ~(size_t)255;
        return at;
    }
};

}  // namespace

cudaError_t build_scene_device(const float* positions_dev, uint32_t num_vertices, const uint32_t* indices_dev,
                               uint32_t num_triangles, const uint32_t* geom_first_dev, uint32_t num_geoms,
                               bool want8, cudaStream_t s, DeviceBuild* out) {
    const uint32_t n = num_triangles;
    if (n < 2 || !out || num_geoms == 0) return cudaErrorInvalidValue;
    *out = DeviceBuild{};
    cudaError_t e = cudaSuccess;
    const size_t ninner = (size_t)n - 1, nall = 2 * (size_t)n - 1;
    const size_t sort_bytes = sort_scratch_bytes(n, 63);
    const int radius = g_ploc_radius;
    // Temporaries in one allocation (an allocation and its release cost
    // 0.05-0.1 ms each; 29 of them were a third of a 3M-triangle build).  The
    // BVH8 nodes are emitted over the sort's and the clustering's buffers,
    // which are dead by then, and copied to their exact size.
    Arena ar;
    const size_t o_keys = ar.take(8 * (size_t)n), o_vals = ar.take(4 * (size_t)n), o_sort = ar.take(sort_bytes);
    const size_t o_boxes = ar.take(32 * nall);
    if (want8) ar.bytes = std::max(ar.bytes, (ninner * sizeof(Bvh8Node) + 255) & ~(size_t)255);
    const size_t o_a = ar.take(4 * (size_t)n), o_b = ar.take(4 * (size_t)n);  // clusters, then emission tasks
    const size_t o_cost = ar.take(want8 ? 32 * ninner : 0), o_meta = ar.take(want8 ? 16 * ninner : 0);
    const size_t ploc_tiles = ((size_t)n + (kBB - 2 * kPlocRMax) - 1) / (kBB - 2 * kPlocRMax);
    const size_t emit_tiles = want8 ? (ninner + kEmitTile - 1) / kEmitTile : 0;
    const size_t o_zero = ar.take(8 * (ploc_tiles + emit_tiles));
    const size_t o_st = ar.take(sizeof(BuildStats));
    unsigned char* tmp = nullptr;
    Bvh2Node* nodes2 = nullptr;
    float4* recs2 = nullptr;
    float4* recs8 = nullptr;
    Bvh8Node* nodes8 = nullptr;
    uint32_t status = 0;
    BuildStats got;

#define WFPT_TRY(x)                      \
    do {                                 \
        if ((e = (x)) != cudaSuccess) goto done; \
    } while (0)

    WFPT_TRY(dev_malloc(reinterpret_cast<void**>(&tmp), ar.bytes));
    WFPT_TRY(dev_malloc(reinterpret_cast<void**>(&nodes2), ninner * sizeof(Bvh2Node)));
    WFPT_TRY(dev_malloc(reinterpret_cast<void**>(&recs2), (size_t)n * sizeof(TriRec)));
    if (want8) WFPT_TRY(dev_malloc(reinterpret_cast<void**>(&recs8), (size_t)n * sizeof(TriRec)));
    {
        uint64_t* keys = reinterpret_cast<uint64_t*>(tmp + o_keys);
        uint32_t* vals = reinterpret_cast<uint32_t*>(tmp + o_vals);
        float4* boxes = reinterpret_cast<float4*>(tmp + o_boxes);
        uint32_t* ids_a = reinterpret_cast<uint32_t*>(tmp + o_a);
        uint32_t* ids_b = reinterpret_cast<uint32_t*>(tmp + o_b);
        float4* cost = reinterpret_cast<float4*>(tmp + o_cost);
        uint4* meta = reinterpret_cast<uint4*>(tmp + o_meta);
        unsigned long long* ploc_state = reinterpret_cast<unsigned long long*>(tmp + o_zero);
        unsigned long long* emit_state = ploc_state + ploc_tiles;
        BuildStats* st = reinterpret_cast<BuildStats*>(tmp + o_st);
        // stage 1: bounds
        BuildStats init;
        std::memset(&init, 0, sizeof(init));
        for (int k = 0; k < 3; ++k) init.bmin[k] = init.cmin[k] = kNone;
        WFPT_TRY(cudaMemcpyAsync(st, &init, sizeof(init), cudaMemcpyHostToDevice, s));
        WFPT_TRY(cudaMemsetAsync(ploc_state, 0, 8 * (ploc_tiles + emit_tiles), s));
        k_tri_bounds<<<blocks(n), kBB, 0, s>>>(positions_dev, num_vertices, indices_dev, n, st);
        // stage 2: keys, sort, leaves
        k_centroid_keys<<<blocks(n), kBB, 0, s>>>(positions_dev, num_vertices, indices_dev, n, st, keys, vals);
        WFPT_TRY(cudaGetLastError());
        WFPT_TRY(launch_sort_pairs(keys, vals, n, nullptr, 63, tmp + o_sort, sort_bytes, s));
        k_leaves<<<blocks(n), kBB, 0, s>>>(vals, n, positions_dev, num_vertices, indices_dev, geom_first_dev,
                                           num_geoms, boxes, recs2, ids_a);
        count_launch(3);
        WFPT_TRY(cudaGetLastError());
        // stage 3: clusters, BVH2, collapse tables
        const float tri_cost = (float)get_bvh8_tri_cost_pct() * 0.01f;
        const uint64_t tile = (uint64_t)(kBB - 2 * radius);
        PlocStart from{n, n, 0, 0};
        for (;;) {
            WFPT_TRY(launch_resident(k_ploc, ((uint64_t)from.clusters + tile - 1) / tile, s, ids_a, ids_b, n, radius,
                                     boxes, reinterpret_cast<float4*>(nodes2), cost, meta, want8 ? 1 : 0, tri_cost,
                                     ploc_state, st, from));
            // stage 4: BVH8
            if (want8)
                WFPT_TRY(launch_resident(k_emit8, (uint64_t)emit_tiles, s, ids_a, ids_b, n, (const Bvh2Node*)nodes2,
                                         (const uint4*)meta, (const float4*)recs2, reinterpret_cast<float4*>(tmp),
                                         recs8, emit_state, st));
            WFPT_TRY(cudaMemcpyAsync(&got, st, sizeof(got), cudaMemcpyDeviceToHost, s));
            WFPT_TRY(cudaStreamSynchronize(s));
            // More passes to go (rare): anything else that left several
            // clusters is an error, seen below.
            if (got.bad_index || got.stuck || got.clusters <= 1 || got.clusters >= from.clusters ||
                got.iterations != from.iterations + kPassesPerLaunch)
                break;
            from = PlocStart{got.clusters, got.next_id, got.iterations, got.pair_ties};
            WFPT_TRY(cudaMemsetAsync(&st->ploc_barrier, 0, sizeof(st->ploc_barrier), s));
        }
    }
    if (got.bad_index) {
        e = cudaErrorInvalidValue;
        goto done;
    }
    out->too_deep = got.too_deep != 0;
    WFPT_TRY(status_build(&status));
    if (status || got.stuck || got.too_deep || got.clusters != 1 || got.next_id != nall || (want8 && got.tris8 != n) ||
        (want8 && (got.nodes8 == 0 || got.nodes8 > ninner))) {
        e = cudaErrorUnknown;
        goto done;
    }
    out->ploc_iterations = got.iterations;
    for (int k = 0; k < 3; ++k) {
        const uint32_t lo = (got.bmin[k] & 0x80000000u) ? (got.bmin[k] & 0x7FFFFFFFu) : ~got.bmin[k];
        const uint32_t hi = (got.bmax[k] & 0x80000000u) ? (got.bmax[k] & 0x7FFFFFFFu) : ~got.bmax[k];
        std::memcpy(&out->bounds_min[k], &lo, 4);
        std::memcpy(&out->bounds_max[k], &hi, 4);
    }
    if (want8) {
        WFPT_TRY(dev_malloc(reinterpret_cast<void**>(&nodes8), got.nodes8 * sizeof(Bvh8Node)));
        WFPT_TRY(cudaMemcpyAsync(nodes8, tmp, got.nodes8 * sizeof(Bvh8Node), cudaMemcpyDeviceToDevice, s));
        WFPT_TRY(cudaStreamSynchronize(s));
        out->bvh8_count = got.nodes8;
    }
    out->bvh2_nodes = nodes2;
    out->bvh2_tris = recs2;
    out->bvh2_count = (uint32_t)ninner;
    out->bvh8_nodes = nodes8;
    out->bvh8_tris = recs8;
    nodes2 = nullptr;
    recs2 = nullptr;
    nodes8 = nullptr;
    recs8 = nullptr;
#undef WFPT_TRY
done:
    for (void* p : {(void*)tmp, (void*)nodes2, (void*)recs2, (void*)recs8, (void*)nodes8})
        if (p) cudaFree(p);
    return e;
}

}  // namespace wfpt
