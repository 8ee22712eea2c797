// Software BVH traversal: replaces trace.comp's rayQuery (trace.comp:50-84)
// on a GPU without RT cores.
//
// Plain form  (WFPT_BVH2_FP32): binary BVH, each 64-byte node holds both
//   children's FP32 boxes; one thread per ray, while-while traversal with a
//   per-thread stack.
// Chosen form (WFPT_BVH8_Q8):   8-wide BVH, 80-byte nodes with an FP32
//   origin, per-axis power-of-two scales and 8-bit child boxes rounded
//   outward; children visited in ray-octant order, node groups on the stack
//   (Ylitie, Karras, Laine: "Efficient Incoherent Ray Traversal on GPUs
//   Through Compressed Wide BVHs", HPG 2017).  Persistent warps: a lane
//   whose ray is done takes the next ray from a global counter (one atomic
//   per warp for all idle lanes), so warps stay full on incoherent rays.
// Both use the watertight ray/triangle test of Woop, Benthin and Wald
// (JCGT 2013), evaluated without FMA contraction, and the same closest-hit
// rule (smallest t, ties to the smaller global triangle index), so both
// forms return identical hits.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "scene.h"
#include "stages.cuh"
#include "trace.cuh"

namespace wfpt {

cudaError_t status_trace(uint32_t* out) { return read_and_clear_status(out); }

constexpr int kStack2 = 64;
constexpr int kStack8 = 32;
// Relative slack on box exit distances (about 2*gamma(3) for FP32).
constexpr float kBoxSlack = 1.0000004f;
constexpr uint32_t kNoRay = 0xFFFFFFFFu;

// Work counters of the counting kernel variants: node visits, triangle
// tests, rays, warp loop iterations (persistent kernel only).
static __device__ unsigned long long g_counts[4];

__device__ __forceinline__ void add_counts(uint32_t nodes, uint32_t tris, uint32_t rays, uint32_t iters) {
    atomicAdd(&g_counts[0], (unsigned long long)nodes);
    atomicAdd(&g_counts[1], (unsigned long long)tris);
    atomicAdd(&g_counts[2], (unsigned long long)rays);
    if (iters) atomicAdd(&g_counts[3], (unsigned long long)iters);
}

struct RayT {
    f3 o;
    f3 inv;
    f3 oinv;  // o * inv
    float tmin;
    int kx, ky, kz;
    float sx, sy, sz;
    uint32_t oct;  // bit k = sign bit of d[k]
    uint32_t perm0, perm1;  // byte c & 3: 1 << (c ^ oct) for the BVH8 slots c = 0..3 and 4..7
};

__device__ __forceinline__ float comp(const f3& v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

__device__ __forceinline__ float safe_inv(float d) {
    const float eps = 1e-20f;
    float a = fabsf(d) > eps ? d : copysignf(eps, d);
    return __fdiv_rn(1.0f, a);
}

__device__ __forceinline__ RayT setup_ray(const float4& r0, const float4& r1) {
    RayT r;
    r.o = mk(r0.x, r0.y, r0.z);
    f3 d = mk(r1.x, r1.y, r1.z);
    r.tmin = r0.w;
    r.inv = mk(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
    r.oinv = mul(r.o, r.inv);
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz + 1 == 3 ? 0 : kz + 1;
    int ky = kx + 1 == 3 ? 0 : kx + 1;
    if (comp(d, kz) < 0.0f) {
        int t = kx;
        kx = ky;
        ky = t;
    }
    r.kx = kx;
    r.ky = ky;
    r.kz = kz;
    float dz = comp(d, kz);
    r.sx = __fdiv_rn(comp(d, kx), dz);
    r.sy = __fdiv_rn(comp(d, ky), dz);
    r.sz = __fdiv_rn(1.0f, dz);
    // Sign bits (not d < 0): -0.0 has a negative reciprocal in safe_inv, and
    // the BVH8 near/far plane choice must agree with the sign of inv.
    r.oct = (__float_as_uint(d.x) >> 31) | ((__float_as_uint(d.y) >> 31) << 1) |
            ((__float_as_uint(d.z) >> 31) << 2);
    const uint32_t low = __byte_perm(0x08040201u, 0u, 0x3210u ^ ((r.oct & 3u) * 0x1111u));
    r.perm0 = low << (r.oct & 4u);
    r.perm1 = low << (4u - (r.oct & 4u));
    return r;
}

// Closest-hit state: distance, tie-break key (global triangle index) and
// the triangle record index; barycentrics are recomputed once at the end.
struct HitS {
    float t;
    uint32_t key;
    uint32_t rec;
};

struct Uvw {
    float U, V, W, det, T;
    bool edge_ok;
};

// Woop-Benthin-Wald edge functions and scaled distance for one triangle,
// from the ray origin, its axis permutation and shear constants.
__device__ __forceinline__ Uvw tri_uvw(const f3& org, int kx, int ky, int kz, float sx, float sy, float sz,
                                       const float4& a4, const float4& b4, const float4& c4) {
    f3 A = sub(mk(a4.x, a4.y, a4.z), org);
    f3 B = sub(mk(b4.x, b4.y, b4.z), org);
    f3 C = sub(mk(c4.x, c4.y, c4.z), org);
    float Akz = comp(A, kz), Bkz = comp(B, kz), Ckz = comp(C, kz);
    float Ax = __fsub_rn(comp(A, kx), __fmul_rn(sx, Akz));
    float Ay = __fsub_rn(comp(A, ky), __fmul_rn(sy, Akz));
    float Bx = __fsub_rn(comp(B, kx), __fmul_rn(sx, Bkz));
    float By = __fsub_rn(comp(B, ky), __fmul_rn(sy, Bkz));
    float Cx = __fsub_rn(comp(C, kx), __fmul_rn(sx, Ckz));
    float Cy = __fsub_rn(comp(C, ky), __fmul_rn(sy, Ckz));
    Uvw q;
    q.U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    q.V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    q.W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (q.U == 0.0f || q.V == 0.0f || q.W == 0.0f) {
        double cxby = (double)Cx * (double)By, cybx = (double)Cy * (double)Bx;
        q.U = (float)(cxby - cybx);
        double axcy = (double)Ax * (double)Cy, aycx = (double)Ay * (double)Cx;
        q.V = (float)(axcy - aycx);
        double bxay = (double)Bx * (double)Ay, byax = (double)By * (double)Ax;
        q.W = (float)(bxay - byax);
    }
    q.edge_ok = !((q.U < 0.0f || q.V < 0.0f || q.W < 0.0f) && (q.U > 0.0f || q.V > 0.0f || q.W > 0.0f));
    q.det = __fadd_rn(__fadd_rn(q.U, q.V), q.W);
    float Az = __fmul_rn(sz, Akz), Bz = __fmul_rn(sz, Bkz), Cz = __fmul_rn(sz, Ckz);
    q.T = __fadd_rn(__fadd_rn(__fmul_rn(q.U, Az), __fmul_rn(q.V, Bz)), __fmul_rn(q.W, Cz));
    return q;
}

__device__ __forceinline__ Uvw tri_uvw(const RayT& r, const float4& a4, const float4& b4, const float4& c4) {
    return tri_uvw(r.o, r.kx, r.ky, r.kz, r.sx, r.sy, r.sz, a4, b4, c4);
}

// Watertight test of record `rec`; on acceptance updates `h`.
__device__ __forceinline__ bool intersect_tri(const RayT& r, const float4* __restrict__ tris, uint32_t rec,
                                              HitS& h) {
    float4 a4 = __ldg(&tris[3 * rec + 0]);
    float4 b4 = __ldg(&tris[3 * rec + 1]);
    float4 c4 = __ldg(&tris[3 * rec + 2]);
    Uvw q = tri_uvw(r, a4, b4, c4);
    if (!q.edge_ok || q.det == 0.0f) return false;
    float t = __fdiv_rn(q.T, q.det);
    if (!(t >= r.tmin)) return false;
    uint32_t key = __float_as_uint(c4.w);
    if (!(t < h.t || (t == h.t && key < h.key))) return false;
    h.t = t;
    h.key = key;
    h.rec = rec;
    return true;
}

// Writes the RayResult of a finished ray (trace.comp:66-84).
__device__ __forceinline__ void write_hit(int4* __restrict__ results, uint32_t ri, const RayT& r,
                                          const float4* __restrict__ tris, const HitS& h, bool found) {
    int4 out;
    if (found) {
        float4 a4 = __ldg(&tris[3 * h.rec + 0]);
        float4 b4 = __ldg(&tris[3 * h.rec + 1]);
        float4 c4 = __ldg(&tris[3 * h.rec + 2]);
        Uvw q = tri_uvw(r, a4, b4, c4);  // same inputs, same edge functions as at acceptance
        float u = __fdiv_rn(q.V, q.det), v = __fdiv_rn(q.W, q.det);
        out = make_int4(__float_as_int(a4.w), __float_as_int(b4.w), __float_as_int(h.t), (int)pack_unorm2x16(u, v));
    } else {
        out = make_int4(-1, -1, __float_as_int(-1.0f), 0);
    }
    results[ri] = out;
}

__device__ __forceinline__ void write_miss(int4* __restrict__ results, uint32_t ri) {
    results[ri] = make_int4(-1, -1, __float_as_int(-1.0f), 0);
}

// ------------------------------------------------------------ BVH2 (plain)
__device__ __forceinline__ void box2(const RayT& r, float lox, float hix, float loy, float hiy, float loz,
                                     float hiz, float tcur, float& tnear, bool& hit) {
    float x0 = __fmaf_rn(lox, r.inv.x, -r.oinv.x), x1 = __fmaf_rn(hix, r.inv.x, -r.oinv.x);
    float y0 = __fmaf_rn(loy, r.inv.y, -r.oinv.y), y1 = __fmaf_rn(hiy, r.inv.y, -r.oinv.y);
    float z0 = __fmaf_rn(loz, r.inv.z, -r.oinv.z), z1 = __fmaf_rn(hiz, r.inv.z, -r.oinv.z);
    float tn = fmaxf(max3f(fminf(x0, x1), fminf(y0, y1), fminf(z0, z1)), r.tmin);
    float tf = fminf(min3f(fmaxf(x0, x1), fmaxf(y0, y1), fmaxf(z0, z1)), tcur);
    tnear = tn;
    hit = tn <= tf * kBoxSlack;
}

// An inner node: goes on to the nearer child hit (the other on the stack) or to
// the top of the stack; false when that is empty.
__device__ __forceinline__ void bvh2_step(const float4* __restrict__ nodes, const RayT& r, float tcur, int& node,
                                          int* stack, int& sp, bool& done) {
    float4 a, b, c, lf;
    load32(nodes + 4 * (size_t)node, a, b);
    load32(nodes + 4 * (size_t)node + 2, c, lf);
    const int2 l = make_int2(__float_as_int(lf.x), __float_as_int(lf.y));
    float t0, t1;
    bool h0, h1;
    box2(r, a.x, a.y, a.z, a.w, c.x, c.y, tcur, t0, h0);
    box2(r, b.x, b.y, b.z, b.w, c.z, c.w, tcur, t1, h1);
    if (h0 && h1) {
        int nearc = l.x, farc = l.y;
        if (t1 < t0) {
            nearc = l.y;
            farc = l.x;
        }
        if (sp < kStack2) {
            stack[sp++] = farc;
        } else {
            raise_status(kErrBounds);
        }
        node = nearc;
    } else if (h0) {
        node = l.x;
    } else if (h1) {
        node = l.y;
    } else if (sp == 0) {
        done = true;
    } else {
        node = stack[--sp];
    }
}

// One ray, traced by one thread.  OCCLUDED: results is an array of words, which
// get 0 for a hit and -1 for a miss.
template <bool CLOSEST, bool COUNT, bool OCCLUDED = false>
__device__ __forceinline__ void trace_bvh2_ray(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                               const float4* __restrict__ rays, int4* __restrict__ results,
                                               uint32_t ri) {
    float4 r0 = rays[2 * ri + 0];
    float4 r1 = rays[2 * ri + 1];
    if (!(r1.w >= r0.w)) {  // tmax < tmin (or NaN): empty interval
        if (OCCLUDED)
            reinterpret_cast<int32_t*>(results)[ri] = -1;
        else
            write_miss(results, ri);
        return;
    }
    RayT r = setup_ray(r0, r1);
    HitS h{r1.w, 0xFFFFFFFFu, 0u};
    bool found = false;
    uint32_t c_nodes = 0, c_tris = 0;
    int stack[kStack2];
    int sp = 0;
    int node = 0;
    bool done = false;
    while (!done) {
        // Inner nodes.
        while (node >= 0) {
            if (COUNT) ++c_nodes;
            bvh2_step(nodes, r, h.t, node, stack, sp, done);
            if (done) break;
        }
        if (done) break;
        // Leaves.
        while (node < 0) {
            uint32_t code = ~(uint32_t)node;
            uint32_t first = code >> 3, cnt = (code & 7u) + 1u;
            for (uint32_t k = 0; k < cnt; ++k) {
                if (COUNT) ++c_tris;
                if (intersect_tri(r, tris, first + k, h)) {
                    found = true;
                    if (!CLOSEST) break;
                }
            }
            if (!CLOSEST && found) {
                done = true;
                break;
            }
            if (sp == 0) {
                done = true;
                break;
            }
            node = stack[--sp];
        }
    }
    if (OCCLUDED)
        reinterpret_cast<int32_t*>(results)[ri] = found ? 0 : -1;
    else
        write_hit(results, ri, r, tris, h, found);
    if (COUNT) add_counts(c_nodes, c_tris, 1u, 0u);
}


// One thread per ray.  Incoherent rays keep 6 to 9 lanes of a warp busy, and
// the kernel waits on its node loads: 66 dependent 64-byte nodes a ray through
// an L1 that is 60 % busy.  So a node is two 256-bit loads instead of four
// 128-bit ones (L1 requests, and with them its busy cycles, fall by a third:
// 2-4 % faster), and wavefronts that fill the GPU run as blocks of two warps
// with registers capped at 51 (20 blocks per SM): a block's registers wait
// for its longest ray, so small blocks keep more warps in flight than
// 256-thread ones.  Closest hit 1773 -> 1648 us (courtyard, 2.07M bounce-1
// rays), 456 -> 423 us (city, 1.6M), camera rays 671 -> 632 and 257 -> 239 us,
// any hit 1679 -> 1569 and 413 -> 387 us; 64 threads without the cap 3-4 %
// slower, with 24 blocks 5-10 %.  Wavefronts below half of the 194,560
// resident rays of that shape gain nothing from it and want the registers
// (57K rays: 161 us in 256-thread blocks, 176 us in small ones; 120K: 186 and
// 173).
constexpr int kBvh2SmallBlock = 64, kBvh2SmallPerSm = 20;
constexpr uint32_t kBvh2SmallMin = 152 * kBvh2SmallPerSm * kBvh2SmallBlock / 2;
template <bool CLOSEST, bool COUNT, int BLOCK, int PER_SM, bool OCCLUDED = false>
__global__ void __launch_bounds__(BLOCK, PER_SM) k_trace_bvh2(const float4* __restrict__ nodes,
                                                              const float4* __restrict__ tris,
                                                              const float4* __restrict__ rays,
                                                              int4* __restrict__ results,
                                                              const uint32_t* __restrict__ ray_index, uint32_t n,
                                                              const uint32_t* __restrict__ n_dev) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= load_count(n, n_dev)) return;
    trace_bvh2_ray<CLOSEST, COUNT, OCCLUDED>(nodes, tris, rays, results, ray_index ? ray_index[i] : i);
}

// The same with resident warps whose lanes take new rays (work[0] hands them
// out; work[1] counts finished warps, and the last resets both), for a
// renderer's bounce and shadow rays.  Incoherent rays take very different
// numbers of steps, and above a warp waits for its longest one with 6 to 9 lanes
// busy.  Here idle lanes get new rays once there are kBvh2Refill of them, and the
// node steps, asked about every fourth time, end when fewer than kBvh2Few lanes
// take one, so that leaves are tested by many lanes at once: 2.07M courtyard
// bounce-1 rays 1648 -> 1220 us, any hit 1567 -> 1399; the city's 1.6M 423 ->
// 344 and 385 -> 304, 6.4M 1462 -> 1186 and 1331 -> 1057.  Rays that go together
// lose by it (camera rays 632 -> 764 and 713 -> 813 us): those keep the kernel
// above, and so do wavefronts smaller than the lanes of this one, which have
// nothing to refill with (262K rays 296 -> 252 us, 228K 278 -> 236, 120K 173 ->
// 189).  It also runs no empty blocks where a bounce's count is far below its
// capacity (68 us at n = 8.3M, 133 us for its shadow rays).  Refill 8, 16, 24,
// 28: 16.4, 15.2, 15.1, 15.9 ms for a 4K city frame that takes 15.1 ms; few 2, 4,
// 10: 15.6, 15.1, 15.2; a vote per step 15.5, every second 15.3; four blocks per
// SM 17.0; two or four leaves in a row 15.6.
//
// It needs counters of the caller's own: a scene's are handed out in turn, and
// two replays of one captured launch at a time would share a pair.
constexpr int kBvh2PerSm = 5;
constexpr unsigned kBvh2Grid = 152 * kBvh2PerSm;
constexpr uint32_t kBvh2RefillMin = 152 * kBvh2PerSm * kBlock;
constexpr int kBvh2Refill = 20, kBvh2Steps = 32, kBvh2Few = 6;
template <bool CLOSEST, bool COUNT, bool OCCLUDED = false>
__global__ void __launch_bounds__(kBlock, kBvh2PerSm) k_trace_bvh2_persistent(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const float4* __restrict__ rays,
    int4* __restrict__ results, const uint32_t* __restrict__ ray_index, uint32_t n,
    const uint32_t* __restrict__ n_dev, uint32_t* __restrict__ work) {
    const uint32_t count = load_count(n, n_dev);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    RayT r;
    HitS h{0.0f, 0xFFFFFFFFu, 0u};
    bool active = false, found = false, exhausted = false;
    uint32_t ri = 0, c_nodes = 0, c_tris = 0, c_rays = 0;
    int stack[kStack2];
    int sp = 0, node = 0;
    for (;;) {
        const bool want = !active && !exhausted;
        const uint32_t want_mask = __ballot_sync(0xffffffffu, want);
        const uint32_t busy_mask = __ballot_sync(0xffffffffu, active);
        if (want_mask != 0u && (__popc(want_mask) >= kBvh2Refill || busy_mask == 0u)) {
            const uint32_t leader = __ffs(want_mask) - 1u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&work[0], __popc(want_mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                const uint32_t i = base + __popc(want_mask & lt_mask);
                if (i < count) {
                    ri = ray_index ? ray_index[i] : i;
                    const float4 r0 = rays[2 * (size_t)ri + 0];
                    const float4 r1 = rays[2 * (size_t)ri + 1];
                    if (!(r1.w >= r0.w)) {  // empty interval: miss, lane stays idle
                        if (OCCLUDED)
                            reinterpret_cast<int32_t*>(results)[ri] = -1;
                        else
                            write_miss(results, ri);
                    } else {
                        r = setup_ray(r0, r1);
                        h = HitS{r1.w, 0xFFFFFFFFu, 0u};
                        active = true;
                        found = false;
                        sp = 0;
                        node = 0;
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, active || !exhausted) == 0u) break;
        // Inner nodes, until few lanes are at one.
        bool done = false;
        for (int st = 0; st < kBvh2Steps; ++st) {
            const bool go = active && !done && node >= 0;
            if ((st & 3) == 3 && __popc(__ballot_sync(0xffffffffu, go)) < kBvh2Few) break;
            if (go) {
                if (COUNT) ++c_nodes;
                bvh2_step(nodes, r, h.t, node, stack, sp, done);
            }
        }
        // A leaf of each lane that has come to one.
        if (active && !done && node < 0) {
            const uint32_t code = ~(uint32_t)node;
            const uint32_t first = code >> 3, cnt = (code & 7u) + 1u;
            for (uint32_t k = 0; k < cnt; ++k) {
                if (COUNT) ++c_tris;
                if (intersect_tri(r, tris, first + k, h)) {
                    found = true;
                    if (!CLOSEST) break;
                }
            }
            if ((!CLOSEST && found) || sp == 0)
                done = true;
            else
                node = stack[--sp];
        }
        if (active && done) {
            if (OCCLUDED)
                reinterpret_cast<int32_t*>(results)[ri] = found ? 0 : -1;
            else
                write_hit(results, ri, r, tris, h, found);
            active = false;
            if (COUNT) ++c_rays;
        }
        __syncwarp();
    }
    if (COUNT) add_counts(c_nodes, c_tris, c_rays, 0u);
    if (lane == 0) {
        const uint32_t warps = gridDim.x * (kBlock / 32);
        __threadfence();
        if (atomicAdd(&work[1], 1u) == warps - 1u) {
            work[0] = 0u;
            work[1] = 0u;
            __threadfence();
        }
    }
}

// --------------------------------------------------------- BVH8 (chosen)
__device__ __forceinline__ uint32_t byte_of(uint32_t w, int b) { return (w >> (8 * b)) & 0xFFu; }

// Byte b of w as the exact float 2^15 + q: one PRMT places the byte in
// mantissa bits 8..15 of 2^15 (bits 0x4700qq00).  The 2^15 bias is folded
// into the node's slab offsets (intersect_node8), so a plane costs one PRMT
// and one FMA.
__device__ __forceinline__ float q2f(uint32_t w, int b) {
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7604u | ((uint32_t)b << 4)));
}
// The same for bytes 0 and 2 by a two-way dot product with 256, off the ALU.
__device__ __forceinline__ float q2f_dot(uint32_t w, int b) {
    return __uint_as_float((b & 2) ? __dp2a_hi(256u, w, 0x47000000u) : __dp2a_lo(256u, w, 0x47000000u));
}

// Two FP32 fused multiply-adds in one instruction (sm_100 and later), each
// rounded as one alone: a child's near and far plane of an axis.
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ void unpair2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// Intersects the eight children of a BVH8 node.  Returns its inner hits in
// bits 24..31 (octant-permuted slot order, highest first) and its leaf hits in
// `leaf` (bit 8 (c & 3) + (c & 4) for slot c), which leaf_count and
// leaf_tris below turn into triangles of the node's second 16 bytes.
// A node step is half of the traversal's time, and bound by issue slots (78 %
// used) and the half-rate ALU pipe (63 %: byte permutes, min/max, selects,
// logic).  So a hit child costs one predicated OR here: shifting its unary
// count to its bit index (two permutes, a shift and an OR per child, and the
// decoding of the meta bytes) is left to the few nodes with leaf hits, once
// per loop iteration, and the inner hits are permuted all at once by two
// 4-way byte dot products: closest hit 1005 -> 949 us (courtyard, 2.07M sorted
// bounce-1 rays), any hit 1221 -> 1141 us.  With the ALU relieved, the paired
// multiply-adds pay too (24 issue slots a node): 949 -> 920 and 1141 -> 1108
// us.  City: 468 -> 444 and 361 -> 339 us.
// DOT: every other byte of an axis by a dot product, for the kernels with
// registers to spare: 65K courtyard rays 105 -> 101 us closest, 84 -> 80 us any
// hit, 57K soup rays 98 -> 95 us.  Under the 64-register cap of the large
// wavefronts' kernels it spills and costs 8 %.
template <bool DOT = false>
__device__ __forceinline__ uint32_t intersect_node8(const float4* __restrict__ nd, const RayT& r, float tcur,
                                                    uint32_t& child_base, uint32_t& imask, uint32_t& leaf) {
    float4 n0 = __ldg(nd + 0);
    float4 n1 = __ldg(nd + 1);
    float4 n2 = __ldg(nd + 2);
    float4 n3 = __ldg(nd + 3);
    float4 n4 = __ldg(nd + 4);
    const uint32_t oct = r.oct;
    uint32_t ew = __float_as_uint(n0.w);
    float scx = __uint_as_float((ew & 0xFFu) << 23);
    float scy = __uint_as_float(((ew >> 8) & 0xFFu) << 23);
    float scz = __uint_as_float(((ew >> 16) & 0xFFu) << 23);
    imask = ew >> 24;
    child_base = __float_as_uint(n1.x);
    // Slab distance = q * (scale*inv) + (p - o) * inv, evaluated as
    // (2^15 + q) * a + (b - 2^15 a).  The folded offset is rounded twice
    // (about 2^-24 * (|b| + 2^15 |a|) each); near planes move earlier and far
    // planes later by m = 2^-7 |a| + 2^-22 |b|, which covers that with room
    // to spare (2^-7 of a quantisation step), so culling stays as
    // conservative as the unfolded form.
    float ax = __fmul_rn(scx, r.inv.x), ay = __fmul_rn(scy, r.inv.y), az = __fmul_rn(scz, r.inv.z);
    const float bx0 = __fmaf_rn(n0.x, r.inv.x, -r.oinv.x);
    const float by0 = __fmaf_rn(n0.y, r.inv.y, -r.oinv.y);
    const float bz0 = __fmaf_rn(n0.z, r.inv.z, -r.oinv.z);
    const float mx = __fmaf_rn(fabsf(bx0), 0x1p-22f, __fmul_rn(fabsf(ax), 0x1p-7f));
    const float my = __fmaf_rn(fabsf(by0), 0x1p-22f, __fmul_rn(fabsf(ay), 0x1p-7f));
    const float mz = __fmaf_rn(fabsf(bz0), 0x1p-22f, __fmul_rn(fabsf(az), 0x1p-7f));
    const float fx0 = __fmaf_rn(-32768.0f, ax, bx0), fy0 = __fmaf_rn(-32768.0f, ay, by0);
    const float fz0 = __fmaf_rn(-32768.0f, az, bz0);
    const float bxn = __fsub_rn(fx0, mx), bxf = __fadd_rn(fx0, mx);
    const float byn = __fsub_rn(fy0, my), byf = __fadd_rn(fy0, my);
    const float bzn = __fsub_rn(fz0, mz), bzf = __fadd_rn(fz0, mz);
    // Near/far planes per axis chosen once per node by the ray octant
    // (d < 0: the hi plane is entered first).
    const bool sx = oct & 1u, sy = oct & 2u, sz = oct & 4u;
    uint32_t nx[2] = {sx ? __float_as_uint(n3.z) : __float_as_uint(n2.x), sx ? __float_as_uint(n3.w) : __float_as_uint(n2.y)};
    uint32_t fx[2] = {sx ? __float_as_uint(n2.x) : __float_as_uint(n3.z), sx ? __float_as_uint(n2.y) : __float_as_uint(n3.w)};
    uint32_t ny[2] = {sy ? __float_as_uint(n4.x) : __float_as_uint(n2.z), sy ? __float_as_uint(n4.y) : __float_as_uint(n2.w)};
    uint32_t fy[2] = {sy ? __float_as_uint(n2.z) : __float_as_uint(n4.x), sy ? __float_as_uint(n2.w) : __float_as_uint(n4.y)};
    uint32_t nz[2] = {sz ? __float_as_uint(n4.z) : __float_as_uint(n3.x), sz ? __float_as_uint(n4.w) : __float_as_uint(n3.y)};
    uint32_t fz[2] = {sz ? __float_as_uint(n3.x) : __float_as_uint(n4.z), sz ? __float_as_uint(n3.y) : __float_as_uint(n4.w)};
    // Pairs {near, far}; children's planes are multiplied and added in pairs.
    const uint64_t A[3] = {pair2(ax, ax), pair2(ay, ay), pair2(az, az)};
    const uint64_t B[3] = {pair2(bxn, bxf), pair2(byn, byf), pair2(bzn, bzf)};
    // Box tests: bit 4 of byte c set for a hit child c.
    uint32_t hit[2] = {0u, 0u};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int w = c >> 2, b = c & 3;
        float tnx, tny, tnz, tfx, tfy, tfz;
        unpair2(fma2(pair2(q2f(nx[w], b), q2f(fx[w], b)), A[0], B[0]), tnx, tfx);
        unpair2(fma2(pair2(q2f(ny[w], b), q2f(fy[w], b)), A[1], B[1]), tny, tfy);
        const bool dot = DOT && (b & 1) == 0;
        const float qn = dot ? q2f_dot(nz[w], b) : q2f(nz[w], b), qf = dot ? q2f_dot(fz[w], b) : q2f(fz[w], b);
        unpair2(fma2(pair2(qn, qf), A[2], B[2]), tnz, tfz);
        float tn = fmaxf(max3f(tnx, tny, tnz), r.tmin);
        float tf = fminf(min3f(tfx, tfy, tfz), tcur);
        if (tn <= tf * kBoxSlack) hit[w] |= 0x10u << (8 * b);
    }
    // Meta bytes: an inner child has bits 5, 4 and 3 set (001 | 24 + slot), a
    // leaf its unary triangle count in bits 5..7 (bit 5 always set) over an
    // offset of at most 23, an empty slot 0.  The inner hits go to their
    // permuted places by the dot product of the 16-valued hit bytes with the
    // ray's bytes 1 << (slot ^ octant).
    const uint32_t m0 = __float_as_uint(n1.z), m1 = __float_as_uint(n1.w);
    const uint32_t in0 = hit[0] & m0 & (m0 << 1), in1 = hit[1] & m1 & (m1 << 1);
    leaf = ((hit[0] & ~in0 & (m0 >> 1)) >> 4) | (hit[1] & ~in1 & (m1 >> 1));
    return __dp4a(in0, r.perm0, __dp4a(in1, r.perm1, 0u)) << 20;
}

// Triangles of a node's leaf hits (`leaf` of intersect_node8), m0 and m1 its
// meta words.
__device__ __forceinline__ uint32_t leaf_count(uint32_t leaf, uint32_t m0, uint32_t m1) {
    return __popc(m0 & ((leaf & 0x01010101u) * 0xE0u)) + __popc(m1 & (((leaf >> 4) & 0x01010101u) * 0xE0u));
}
// The same as bits 0..23 relative to the node's first triangle.
__device__ __forceinline__ uint32_t leaf_tris(uint32_t leaf, uint32_t m0, uint32_t m1) {
    uint32_t tris = 0;
    while (leaf != 0u) {
        const uint32_t bit = (uint32_t)__ffs(leaf) - 1u;
        leaf &= leaf - 1u;
        const uint32_t m = ((bit & 4u) ? m1 : m0) >> (bit & 24u);
        tris |= ((m >> 5) & 7u) << (m & 31u);
    }
    return tris;
}

// Persistent-warp traversal.  work[0] = next ray to hand out, work[1] =
// warps finished; the last warp to finish resets both, so the counters
// need no reset between launches that use them one after another.
template <bool CLOSEST, bool COUNT>
__global__ void __launch_bounds__(kBlock, 4) k_trace_bvh8(const float4* __restrict__ nodes,
                                                          const float4* __restrict__ tris,
                                                          const float4* __restrict__ rays, int4* __restrict__ results,
                                                          const uint32_t* __restrict__ ray_index, uint32_t n,
                                                          const uint32_t* __restrict__ n_dev,
                                                          uint32_t* __restrict__ work, uint32_t refill, uint32_t postpone) {
    const uint32_t count = load_count(n, n_dev);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint2 stack[kStack8];
    int sp = 0;
    uint32_t ri = kNoRay;
    // Lane state: idle (no ray), tracing, or done (result held in registers
    // until the next refill of the warp writes it, so the divergent write-out
    // runs once per refill instead of once per finished ray).
    enum : uint32_t { kIdle = 0, kTracing = 1, kDone = 2 };
    uint32_t state = kIdle;
    bool exhausted = false, found = false;
    RayT r;
    HitS h;
    uint2 ng = make_uint2(0u, 0u);  // node group: child base, hit bits 24..31 | imask 0..7
    uint32_t c_nodes = 0, c_tris = 0, c_rays = 0, c_iters = 0;
    for (;;) {
        // Refill non-tracing lanes with new rays (one atomic per warp).
        bool want = state != kTracing && !exhausted;
        uint32_t want_mask = __ballot_sync(0xffffffffu, want);
        uint32_t busy_mask = __ballot_sync(0xffffffffu, state == kTracing);
        if (want_mask != 0u && (__popc(want_mask) >= refill || busy_mask == 0u)) {
            if (state == kDone) {
                write_hit(results, ri, r, tris, h, found);
                state = kIdle;
            }
            uint32_t leader = __ffs(want_mask) - 1u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&work[0], __popc(want_mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                uint32_t i = base + __popc(want_mask & lt_mask);
                if (i < count) {
                    uint32_t idx = ray_index ? ray_index[i] : i;
                    float4 r0 = rays[2 * idx + 0];
                    float4 r1 = rays[2 * idx + 1];
                    if (!(r1.w >= r0.w)) {  // empty interval: miss, lane stays idle
                        write_miss(results, idx);
                    } else {
                        ri = idx;
                        state = kTracing;
                        r = setup_ray(r0, r1);
                        h = HitS{r1.w, 0xFFFFFFFFu, 0u};
                        found = false;
                        sp = 0;
                        ng = make_uint2(0u, 0x80000000u);  // root as the only child of a virtual group
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        const uint32_t busy = __ballot_sync(0xffffffffu, state == kTracing);
        if (__ballot_sync(0xffffffffu, state != kIdle || !exhausted) == 0u) break;
        if (COUNT && lane == 0) ++c_iters;
        if (state != kTracing) continue;

        // The current group is either a node group (hit bits 24..31) or a
        // triangle group popped from the stack (bits 0..23, base in x).
        uint32_t tri_base = 0, tg = 0;
        if (ng.y > 0x00FFFFFFu) {
            // One node: pick the nearest child of the current group.
            uint32_t bit = 31u - __clz(ng.y);
            ng.y &= ~(1u << bit);
            uint32_t slot = (bit - 24u) ^ r.oct;
            uint32_t node = ng.x + __popc(ng.y & ((1u << slot) - 1u) & 0xFFu);
            if (ng.y > 0x00FFFFFFu) {
                if (sp < kStack8) {
                    stack[sp++] = ng;
                } else {
                    raise_status(kErrBounds);
                }
            }
            uint32_t child_base, imask, leaf;
            if (COUNT) ++c_nodes;
            const float4* nd = nodes + 5 * (size_t)node;
            const uint32_t inner = intersect_node8(nd, r, h.t, child_base, imask, leaf);
            ng = make_uint2(child_base, inner | imask);
            if (leaf != 0u) {
                const float4 n1 = __ldg(nd + 1);
                tri_base = __float_as_uint(n1.y);
                tg = leaf_tris(leaf, __float_as_uint(n1.z), __float_as_uint(n1.w));
            }
        } else {
            tri_base = ng.x;
            tg = ng.y;
            ng = make_uint2(0u, 0u);
        }
        // Postpone a node's triangles while few lanes of the warp have any
        // and more nodes remain: they wait on the stack as a triangle group.
        if (postpone != 0u) {
            uint32_t with_tris = __ballot_sync(busy, tg != 0u);
            if (tg != 0u && ng.y > 0x00FFFFFFu && (uint32_t)__popc(with_tris) < postpone && sp < kStack8) {
                stack[sp++] = make_uint2(tri_base, tg);
                tg = 0;
            }
        }
        bool finished = false;
        while (tg != 0u) {
            uint32_t tb = __ffs(tg) - 1u;
            tg &= tg - 1u;
            if (COUNT) ++c_tris;
            if (intersect_tri(r, tris, tri_base + tb, h)) {
                found = true;
                if (!CLOSEST) {
                    finished = true;
                    break;
                }
            }
        }
        if (!finished && ng.y <= 0x00FFFFFFu) {
            if (sp == 0) {
                finished = true;
            } else {
                ng = stack[--sp];
            }
        }
        if (finished) {
            state = kDone;
            if (COUNT) ++c_rays;
        }
    }
    if (COUNT) add_counts(c_nodes, c_tris, c_rays, c_iters);
    // Last warp out resets the work counters for the next launch.
    if (lane == 0) {
        uint32_t warps = gridDim.x * (blockDim.x / 32);
        __threadfence();
        if (atomicAdd(&work[1], 1u) == warps - 1u) {
            work[0] = 0u;
            work[1] = 0u;
            __threadfence();
        }
    }
}

// ------------------------------------ BVH8 with warp-cooperative triangles
// Ray fields the triangle test reads, kept in shared memory so that any
// lane of the warp can test a triangle against any other lane's ray.
struct alignas(16) RayS {
    float ox, oy, oz, tmin;
    float sx, sy, sz;
    uint32_t k;  // kx | ky << 2 | kz << 4
};

__device__ __forceinline__ RayS ray_shared(const RayT& r) {
    RayS s;
    s.ox = r.o.x;
    s.oy = r.o.y;
    s.oz = r.o.z;
    s.tmin = r.tmin;
    s.sx = r.sx;
    s.sy = r.sy;
    s.sz = r.sz;
    s.k = (uint32_t)r.kx | ((uint32_t)r.ky << 2) | ((uint32_t)r.kz << 4);
    return s;
}

__device__ __forceinline__ Uvw tri_uvw(const RayS& s, const float4& a4, const float4& b4, const float4& c4) {
    return tri_uvw(mk(s.ox, s.oy, s.oz), (int)(s.k & 3u), (int)((s.k >> 2) & 3u), (int)(s.k >> 4), s.sx, s.sy, s.sz,
                   a4, b4, c4);
}

// The closest-hit order as one 64-bit key: distance bits mapped to an
// order-preserving unsigned (-0 folded onto +0, so equal distances compare
// equal), then the global triangle index.  atomicMin over these keys picks
// the hit of the sequential rule (smaller t, then smaller index) in any
// order of arrival.
__device__ __forceinline__ unsigned long long hit_key(float t, uint32_t key) {
    uint32_t b = __float_as_uint(__fadd_rn(t, 0.0f));
    b ^= (uint32_t)((int32_t)b >> 31) | 0x80000000u;
    return ((unsigned long long)b << 32) | key;
}

// Any-hit order: pairs of the first group that a loop iteration handed the
// lane before those of the second, then the closest-hit order (triangle
// indices are below 2^27).
__device__ __forceinline__ unsigned long long any_key(float t, uint32_t key, bool second) {
    return ((unsigned long long)second << 60) | ((hit_key(t, 0u) >> 32) << 28) | key;
}

__device__ __forceinline__ float hit_key_t(unsigned long long k) {
    uint32_t b = (uint32_t)(k >> 32);
    b = (b & 0x80000000u) ? (b ^ 0x80000000u) : ~b;
    return __uint_as_float(b);
}

constexpr uint32_t kRecBits = 27;  // task word: lane << 27 | triangle record
constexpr int kRing = 1024;        // per-warp ring of pending triangle tests (power of two)

// Same traversal as k_trace_bvh8, except that triangle tests are shared by
// the warp: each node step appends its lanes' (lane, triangle) pairs to a
// ring in shared memory, and the warp tests the ring 32 pairs at a time,
// each result folded into the owner's best hit key with a shared atomicMin;
// the test whose key is the owner's best after its round stores the hit's
// primitive, geometry, barycentrics and t beside it, so a finished lane
// writes its RayResult from shared memory (no reload of the winning
// triangle at write-out: 2 % faster any hit).  Tests are batched across node
// steps: the ring is tested once `batch` or more pairs are pending (in whole
// passes of 32 when 32 or more are), and entirely once the lanes waiting on
// their own tests plus the idle lanes would fill a refill, or no lane has
// nodes left.  A loop iteration takes up to `steps` node steps per lane, so
// the per-iteration work (refill check, votes, scan, test decision) is shared
// by several node steps.  A lane's ray finishes only when its traversal is
// exhausted (any hit: when it has a hit) and all of its own tests have run,
// so a ring entry never outlives its ray.  The deferred tests leave tcur
// larger for a few node steps (culling stays conservative: tcur only
// shrinks), which costs about 1 % more node steps and saves most of the
// partly empty test passes (batch 1: test every step).
//
// The node steps of an iteration are where lanes sit idle, and they are half
// of the time: a lane that stopped at its first triangles waited for the rest
// of the iteration, so more than two (any hit: three) steps did not pay.  A
// lane now goes on with its triangles in hand until a second node hands it
// some (or the first handed it more than kMoreLeaves leaves), and four steps do:
// closest hit 1070 -> 1003 us (courtyard, 2.07M sorted bounce-1 rays), 502 ->
// 467 us (city, 1.6M), 122 -> 104 us (57K rays of the 65K soup); any hit
// 1286 -> 1221, 393 -> 361 and 119 -> 109 us.  A closest-hit iteration asks
// once, before its third step, whether any lane goes on (a vote per step cost
// 0.3 %, none 0.6 %).  An any-hit iteration ends as soon as fewer than
// kFewLanes lanes go on while there are rays to refill with: its rays are
// short, and an early end brings the refill forward (city 392 -> 361 us
// against steps taken to the end; a share of the tracing lanes instead of a
// number 396-421, 16 or 22 lanes 362-363, 18 lanes and six steps 375).
// A lane appends at most 3 kMoreLeaves + 24 triangles per iteration, so at most
// 31 + 32 * 30 pairs are pending after an append: they fit the ring.
constexpr uint32_t kMoreLeaves = 2;
constexpr uint32_t kFewLanes = 20;
constexpr uint32_t kCoopLargeMin = 4 * 152 * 4 * kBlock;  // wavefronts of the four-block form
static_assert(31 + 32 * (3 * kMoreLeaves + 24) <= kRing, "the ring holds every pending pair");

// PER_SM: four blocks per SM (64 registers) keep the GPU busy on large
// wavefronts; a small one is bound by the latency of its longest rays, and
// three blocks per SM (80 registers) make each step shorter: 57K soup rays
// 104 -> 100 us closest, 120K courtyard rays 150 -> 135, 262K 215 -> 203; any
// hit 105 -> 91 us at 131K rays, 209 -> 206 at 524K.  Even at about 620K rays
// (four times the rays resident at once), 2-4 % slower at 1M, 5 % at 2M; two
// blocks per SM are equal to three below 120K rays and slower above.  Small
// wavefronts that share the GPU (batched requests on several branches) keep
// the four-block form: a 12-request batch 23.6 ms, 24.0 with three.
template <bool CLOSEST, bool COUNT, int PER_SM>
__global__ void __launch_bounds__(kBlock, PER_SM) k_trace_bvh8_coop(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const float4* __restrict__ rays,
    int4* __restrict__ results, const uint32_t* __restrict__ ray_index, uint32_t n,
    const uint32_t* __restrict__ n_dev, uint32_t* __restrict__ work,
    uint32_t refill, uint32_t batch, uint32_t steps) {
    __shared__ RayS s_ray[kBlock];
    __shared__ unsigned long long s_best[kBlock];
    __shared__ uint4 s_hit[kBlock];  // winning hit: primId, geomId, packed barycentrics, t
    __shared__ uint32_t s_task[kBlock / 32][kRing];
    __shared__ float s_tmax[CLOSEST ? 1 : kBlock];       // any hit: the ray's tmax
    __shared__ uint32_t s_second[CLOSEST ? 1 : kBlock];  // any hit: where the lane's second group starts in the ring
    const uint32_t count = load_count(n, n_dev);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t wbase = threadIdx.x & ~31u;
    uint32_t* const task = s_task[threadIdx.x >> 5];
    uint2 stack[kStack8];
    int sp = 0;
    uint32_t ri = kNoRay;
    enum : uint32_t { kIdle = 0, kTracing = 1, kDone = 2 };
    uint32_t state = kIdle;
    bool exhausted = false;
    RayT r;
    float tcur = 0.0f;
    uint2 ng = make_uint2(0u, 0u);
    // Ring counters (absolute, wrapped by the ring mask; equal in all
    // lanes): pairs [tested, appended) are pending.  my_end: one past this
    // lane's last appended pair.
    uint32_t tested = 0, appended = 0, my_end = 0;
    uint32_t c_nodes = 0, c_tris = 0, c_rays = 0, c_iters = 0;
    for (;;) {
        bool want = state != kTracing && !exhausted;
        uint32_t want_mask = __ballot_sync(0xffffffffu, want);
        uint32_t busy_mask = __ballot_sync(0xffffffffu, state == kTracing);
        if (want_mask != 0u && (__popc(want_mask) >= refill || busy_mask == 0u)) {
            if (state == kDone) {
                const unsigned long long best = s_best[threadIdx.x];
                if (CLOSEST ? (uint32_t)best == 0xFFFFFFFFu : best == ~0ull) {
                    write_miss(results, ri);
                } else {
                    const uint4 hh = s_hit[threadIdx.x];
                    results[ri] = make_int4((int)hh.x, (int)hh.y, (int)hh.w, (int)hh.z);
                }
                state = kIdle;
            }
            uint32_t leader = __ffs(want_mask) - 1u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&work[0], __popc(want_mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                uint32_t i = base + __popc(want_mask & lt_mask);
                if (i < count) {
                    uint32_t idx = ray_index ? ray_index[i] : i;
                    float4 r0 = rays[2 * idx + 0];
                    float4 r1 = rays[2 * idx + 1];
                    if (!(r1.w >= r0.w)) {  // empty interval: miss, lane stays idle
                        write_miss(results, idx);
                    } else {
                        ri = idx;
                        state = kTracing;
                        r = setup_ray(r0, r1);
                        s_ray[threadIdx.x] = ray_shared(r);
                        s_best[threadIdx.x] = CLOSEST ? hit_key(r1.w, 0xFFFFFFFFu) : ~0ull;
                        if (!CLOSEST) s_tmax[threadIdx.x] = r1.w;
                        tcur = r1.w;
                        sp = 0;
                        ng = make_uint2(0u, 0x80000000u);
                    }
                } else {
                    exhausted = true;
                }
            }
            want_mask = 0u;  // refilled (or out of rays)
        }
        if (__ballot_sync(0xffffffffu, state != kIdle || !exhausted) == 0u) break;
        if (COUNT && lane == 0) ++c_iters;

        // Up to `steps` node steps, with up to two nodes' leaf hits in hand.
        uint32_t leaf = 0, leaf2 = 0, from = 0, from2 = 0;
        const uint32_t few = CLOSEST ? 0u : (__any_sync(0xffffffffu, exhausted) ? 1u : kFewLanes);
        for (uint32_t st = 0; st < steps; ++st) {
            const bool go = state == kTracing && ng.y > 0x00FFFFFFu && leaf2 == 0u && __popc(leaf) <= kMoreLeaves;
            if (CLOSEST ? (st == 2u && !__any_sync(0xffffffffu, go))
                        : (st >= 1u && (uint32_t)__popc(__ballot_sync(0xffffffffu, go)) < few))
                break;
            if (go) {
                uint32_t bit = 31u - __clz(ng.y);
                ng.y &= ~(1u << bit);
                uint32_t slot = (bit - 24u) ^ r.oct;
                uint32_t node = ng.x + __popc(ng.y & ((1u << slot) - 1u) & 0xFFu);
                if (ng.y > 0x00FFFFFFu) {
                    if (sp < kStack8) {
                        stack[sp++] = ng;
                    } else {
                        raise_status(kErrBounds);
                    }
                }
                uint32_t child_base, imask, lf;
                if (COUNT) ++c_nodes;
                const uint32_t inner = intersect_node8<PER_SM == 3>(nodes + 5 * (size_t)node, r, tcur, child_base, imask, lf);
                ng = make_uint2(child_base, inner | imask);
                if (leaf == 0u) {
                    leaf = lf;
                    from = node;
                } else {
                    leaf2 = lf;
                    from2 = node;
                }
            }
            if (state == kTracing && ng.y <= 0x00FFFFFFu && sp > 0) ng = stack[--sp];
        }

        // Append the pairs: exclusive scan of the per-lane counts.  The nodes'
        // meta words and first triangles are read again here, mostly from
        // L1, by the lanes with leaf hits.
        uint4 meta = make_uint4(0u, 0u, 0u, 0u), meta2 = meta;
        if (leaf != 0u) meta = __ldg(reinterpret_cast<const uint4*>(nodes + 5 * (size_t)from + 1));
        if (leaf2 != 0u) meta2 = __ldg(reinterpret_cast<const uint4*>(nodes + 5 * (size_t)from2 + 1));
        const uint32_t cnt1 = leaf_count(leaf, meta.z, meta.w);
        const uint32_t cnt = cnt1 + leaf_count(leaf2, meta2.z, meta2.w);
        uint32_t incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (cnt != 0u) {
            uint32_t pos = appended + incl - cnt;
            const uint32_t owner = lane << kRecBits;
            if (!CLOSEST) s_second[threadIdx.x] = pos + cnt1;
            while (leaf != 0u) {
                const uint32_t bit = (uint32_t)__ffs(leaf) - 1u;
                leaf &= leaf - 1u;
                const uint32_t m = ((bit & 4u) ? meta.w : meta.z) >> (bit & 24u);
                const uint32_t w = owner | (meta.y + (m & 31u));
                task[pos++ & (kRing - 1)] = w;
                if (m & 0x40u) task[pos++ & (kRing - 1)] = w + 1u;
                if (m & 0x80u) task[pos++ & (kRing - 1)] = w + 2u;
                if (leaf == 0u) {
                    leaf = leaf2;
                    meta = meta2;
                    leaf2 = 0u;
                }
            }
            my_end = pos;
            if (COUNT) c_tris += cnt;
        }
        appended += total;

        // A tracing lane without nodes left waits for its own tests.
        const bool waiting = state == kTracing && ng.y <= 0x00FFFFFFu;
        const uint32_t walk_mask = __ballot_sync(0xffffffffu, state == kTracing && !waiting);
        const uint32_t wait_mask = __ballot_sync(0xffffffffu, waiting && (int32_t)(my_end - tested) > 0);
        const uint32_t pend = appended - tested;
        uint32_t nflush = 0;
        if (pend != 0u) {
            if (walk_mask == 0u || batch <= 1u || (uint32_t)__popc(wait_mask | want_mask) >= refill)
                nflush = pend;
            else if (pend >= batch)
                nflush = pend >= 32u ? (pend & ~31u) : pend;
        }
        if (nflush != 0u) {
            __syncwarp();
            for (uint32_t j0 = 0; j0 < nflush; j0 += 32u) {
                const uint32_t j = j0 + lane;
                bool cand = false;
                unsigned long long hk = 0;
                uint32_t o = 0;
                uint4 hh = make_uint4(0u, 0u, 0u, 0u);
                if (j < nflush) {
                    const uint32_t w = task[(tested + j) & (kRing - 1)];
                    o = wbase + (w >> kRecBits);
                    const uint32_t rec = w & ((1u << kRecBits) - 1u);
                    const RayS rs = s_ray[o];
                    float4 a4 = __ldg(&tris[3 * rec + 0]);
                    float4 b4 = __ldg(&tris[3 * rec + 1]);
                    float4 c4 = __ldg(&tris[3 * rec + 2]);
                    Uvw q = tri_uvw(rs, a4, b4, c4);
                    if (q.edge_ok && q.det != 0.0f) {
                        float t = __fdiv_rn(q.T, q.det);
                        if (t >= rs.tmin && (CLOSEST || t <= s_tmax[o])) {
                            // A stale read can only be larger than the current
                            // best, so skipping on it is safe.
                            hk = CLOSEST ? hit_key(t, __float_as_uint(c4.w))
                                         : any_key(t, __float_as_uint(c4.w), (int32_t)(tested + j - s_second[o]) >= 0);
                            if (hk < s_best[o]) {
                                atomicMin(&s_best[o], hk);
                                cand = true;
                                const float u = __fdiv_rn(q.V, q.det), v = __fdiv_rn(q.W, q.det);
                                hh = make_uint4(__float_as_uint(a4.w), __float_as_uint(b4.w), pack_unorm2x16(u, v),
                                                __float_as_uint(t));
                            }
                        }
                    }
                }
                // The candidate whose key is the owner's best after this
                // round records the hit's fields (keys are unique).
                __syncwarp();
                if (cand && s_best[o] == hk) s_hit[o] = hh;
            }
            __syncwarp();
            tested += nflush;
        }

        if (state == kTracing) {
            const unsigned long long best = s_best[threadIdx.x];
            if (CLOSEST) tcur = hit_key_t(best);
            bool stop = waiting;
            if (!CLOSEST && best != ~0ull) {
                stop = true;  // any hit: no more node steps
                ng.y = 0u;
                sp = 0;
            }
            if (stop && (int32_t)(my_end - tested) <= 0) {
                state = kDone;
                if (COUNT) ++c_rays;
            }
        }
    }
    if (COUNT) add_counts(c_nodes, c_tris, c_rays, c_iters);
    if (lane == 0) {
        uint32_t warps = gridDim.x * (blockDim.x / 32);
        __threadfence();
        if (atomicAdd(&work[1], 1u) == warps - 1u) {
            work[0] = 0u;
            work[1] = 0u;
            __threadfence();
        }
    }
}

// Any-hit traversal: that of k_trace_bvh8_coop for rays that are tested after
// every iteration (its batch 1, the default).  Then a lane has nothing to wait
// for, and the pairs need no ring: 2.07M courtyard bounce-1 hits (two rays
// each) 1108 -> 1091 us, the city's 1.6M 339 -> 330, 6.4M 1245 -> 1211.
//
// !RECORD: for occlusion alone.  A shadow pass reads no more of a hit than that
// there is one, so any accepted triangle will do: no keys and atomics, no order
// among the triangles in hand, no barycentrics, and one word per ray (0, or -1
// if nothing is in the way) instead of sixteen bytes.  The nine shadow passes
// of a 1080p courtyard frame (two rays per hit) 10.11 -> 9.02 ms, reading them
// back 0.51 -> 0.45 ms.  The nearest child first is best here too (1040 us
// against 1081 in slot order and 1098 farthest first; the city 314, 311, 309).
// Small wavefronts (PER_SM 3) go on past four leaves: 256x256 frame 914 -> 893
// us; large ones that way 0.6 % slower.
constexpr uint32_t kFewOccluded = 16;  // 20: 0-1 % slower, 24: 1-3 %, 12: 0-1 %
template <bool RECORD, int PER_SM, bool COUNT = false>
__global__ void __launch_bounds__(kBlock, PER_SM) k_any_bvh8(
    const float4* __restrict__ nodes, const float4* __restrict__ tris, const float4* __restrict__ rays,
    void* __restrict__ results, const uint32_t* __restrict__ ray_index, uint32_t n,
    const uint32_t* __restrict__ n_dev, uint32_t* __restrict__ work, uint32_t refill, uint32_t steps) {
    __shared__ RayS s_ray[kBlock];
    __shared__ float s_tmax[kBlock];
    __shared__ uint32_t s_hit[RECORD ? 1 : kBlock];
    __shared__ unsigned long long s_best[RECORD ? kBlock : 1];
    __shared__ uint4 s_rec[RECORD ? kBlock : 1];        // best hit: primId, geomId, packed barycentrics, t
    __shared__ uint32_t s_second[RECORD ? kBlock : 1];  // where the pairs of the lane's second group start
    constexpr uint32_t MORE = !RECORD && PER_SM == 3 ? 4u : kMoreLeaves;
    __shared__ uint32_t s_task[kBlock / 32][32 * (3 * MORE + 24)];
    const uint32_t count = load_count(n, n_dev);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t wbase = threadIdx.x & ~31u;
    uint32_t* const task = s_task[threadIdx.x >> 5];
    uint2 stack[kStack8];
    int sp = 0;
    uint32_t ri = kNoRay;
    enum : uint32_t { kIdle = 0, kTracing = 1, kFree = 2, kBlocked = 3 };
    uint32_t state = kIdle;
    bool exhausted = false;
    RayT r;
    float tmax = 0.0f;
    uint2 ng = make_uint2(0u, 0u);
    uint32_t c_nodes = 0, c_tris = 0, c_rays = 0, c_iters = 0;
    for (;;) {
        const bool want = state != kTracing && !exhausted;
        const uint32_t want_mask = __ballot_sync(0xffffffffu, want);
        const uint32_t busy_mask = __ballot_sync(0xffffffffu, state == kTracing);
        if (want_mask != 0u && (__popc(want_mask) >= refill || busy_mask == 0u)) {
            if (state >= kFree) {
                if (!RECORD) {
                    static_cast<int32_t*>(results)[ri] = state == kBlocked ? 0 : -1;
                } else if (state == kBlocked) {
                    const uint4 h = s_rec[threadIdx.x];
                    static_cast<int4*>(results)[ri] = make_int4((int)h.x, (int)h.y, (int)h.w, (int)h.z);
                } else {
                    write_miss(static_cast<int4*>(results), ri);
                }
                state = kIdle;
            }
            const uint32_t leader = __ffs(want_mask) - 1u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&work[0], __popc(want_mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (want) {
                const uint32_t i = base + __popc(want_mask & lt_mask);
                if (i < count) {
                    const uint32_t idx = ray_index ? ray_index[i] : i;
                    const float4 r0 = rays[2 * (size_t)idx + 0];
                    const float4 r1 = rays[2 * (size_t)idx + 1];
                    if (!(r1.w >= r0.w)) {  // empty interval: nothing in the way, lane stays idle
                        if (RECORD)
                            write_miss(static_cast<int4*>(results), idx);
                        else
                            static_cast<int32_t*>(results)[idx] = -1;
                    } else {
                        ri = idx;
                        state = kTracing;
                        r = setup_ray(r0, r1);
                        s_ray[threadIdx.x] = ray_shared(r);
                        s_tmax[threadIdx.x] = r1.w;
                        if (RECORD)
                            s_best[threadIdx.x] = ~0ull;
                        else
                            s_hit[threadIdx.x] = 0u;
                        tmax = r1.w;
                        sp = 0;
                        ng = make_uint2(0u, 0x80000000u);
                    }
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, state != kIdle || !exhausted) == 0u) break;
        if (COUNT && lane == 0) ++c_iters;

        uint32_t leaf = 0, leaf2 = 0, from = 0, from2 = 0;
        const uint32_t few = __any_sync(0xffffffffu, exhausted) ? 1u : RECORD ? kFewLanes : kFewOccluded;
        for (uint32_t st = 0; st < steps; ++st) {
            const bool go = state == kTracing && ng.y > 0x00FFFFFFu && leaf2 == 0u && __popc(leaf) <= MORE;
            if (st >= 1u && (uint32_t)__popc(__ballot_sync(0xffffffffu, go)) < few) break;
            if (go) {
                const uint32_t bit = 31u - __clz(ng.y);
                ng.y &= ~(1u << bit);
                const uint32_t slot = (bit - 24u) ^ r.oct;
                const uint32_t node = ng.x + __popc(ng.y & ((1u << slot) - 1u) & 0xFFu);
                if (ng.y > 0x00FFFFFFu) {
                    if (sp < kStack8) {
                        stack[sp++] = ng;
                    } else {
                        raise_status(kErrBounds);
                    }
                }
                uint32_t child_base, imask, lf;
                if (COUNT) ++c_nodes;
                const uint32_t inner = intersect_node8<PER_SM == 3>(nodes + 5 * (size_t)node, r, tmax, child_base, imask, lf);
                ng = make_uint2(child_base, inner | imask);
                if (leaf == 0u) {
                    leaf = lf;
                    from = node;
                } else {
                    leaf2 = lf;
                    from2 = node;
                }
            }
            if (state == kTracing && ng.y <= 0x00FFFFFFu && sp > 0) ng = stack[--sp];
        }

        // The iteration's pairs, at an exclusive scan of the per-lane counts.
        uint4 meta = make_uint4(0u, 0u, 0u, 0u), meta2 = meta;
        if (leaf != 0u) meta = __ldg(reinterpret_cast<const uint4*>(nodes + 5 * (size_t)from + 1));
        if (leaf2 != 0u) meta2 = __ldg(reinterpret_cast<const uint4*>(nodes + 5 * (size_t)from2 + 1));
        const uint32_t cnt1 = leaf_count(leaf, meta.z, meta.w);
        const uint32_t cnt = cnt1 + leaf_count(leaf2, meta2.z, meta2.w);
        if (COUNT) c_tris += cnt;
        uint32_t incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (total != 0u) {
            uint32_t pos = incl - cnt;
            const uint32_t owner = lane << kRecBits;
            if (RECORD) s_second[threadIdx.x] = pos + cnt1;
            while (leaf != 0u) {
                const uint32_t bit = (uint32_t)__ffs(leaf) - 1u;
                leaf &= leaf - 1u;
                const uint32_t m = ((bit & 4u) ? meta.w : meta.z) >> (bit & 24u);
                const uint32_t w = owner | (meta.y + (m & 31u));
                task[pos++] = w;
                if (m & 0x40u) task[pos++] = w + 1u;
                if (m & 0x80u) task[pos++] = w + 2u;
                if (leaf == 0u) {
                    leaf = leaf2;
                    meta = meta2;
                    leaf2 = 0u;
                }
            }
            __syncwarp();
            for (uint32_t j0 = 0; j0 < total; j0 += 32u) {
                const uint32_t j = j0 + lane;
                uint32_t o = 0;
                bool cand = false;
                unsigned long long hk = 0;
                uint4 h = make_uint4(0u, 0u, 0u, 0u);
                if (j < total) {
                    const uint32_t w = task[j];
                    o = wbase + (w >> kRecBits);
                    const uint32_t rec = w & ((1u << kRecBits) - 1u);
                    const RayS rs = s_ray[o];
                    const float4 a4 = __ldg(&tris[3 * rec + 0]), b4 = __ldg(&tris[3 * rec + 1]);
                    const float4 c4 = __ldg(&tris[3 * rec + 2]);
                    const Uvw q = tri_uvw(rs, a4, b4, c4);
                    if (q.edge_ok && q.det != 0.0f) {
                        const float t = __fdiv_rn(q.T, q.det);
                        if (t >= rs.tmin && t <= s_tmax[o]) {
                            if (!RECORD) {
                                s_hit[o] = 1u;
                            } else {
                                hk = any_key(t, __float_as_uint(c4.w), j >= s_second[o]);
                                if (hk < s_best[o]) {  // a stale read can only be larger
                                    atomicMin(&s_best[o], hk);
                                    cand = true;
                                    const float u = __fdiv_rn(q.V, q.det), v = __fdiv_rn(q.W, q.det);
                                    h = make_uint4(__float_as_uint(a4.w), __float_as_uint(b4.w), pack_unorm2x16(u, v),
                                                   __float_as_uint(t));
                                }
                            }
                        }
                    }
                }
                if (RECORD) {  // the best of the round records its fields (keys are unique)
                    __syncwarp();
                    if (cand && s_best[o] == hk) s_rec[o] = h;
                }
            }
            __syncwarp();
        }
        if (state == kTracing) {
            if (RECORD ? s_best[threadIdx.x] != ~0ull : s_hit[threadIdx.x] != 0u)
                state = kBlocked;
            else if (ng.y <= 0x00FFFFFFu)
                state = kFree;
            if (COUNT && state != kTracing) ++c_rays;
        }
    }
    if (COUNT) add_counts(c_nodes, c_tris, c_rays, c_iters);
    if (lane == 0) {
        const uint32_t warps = gridDim.x * (blockDim.x / 32);
        __threadfence();
        if (atomicAdd(&work[1], 1u) == warps - 1u) {
            work[0] = 0u;
            work[1] = 0u;
            __threadfence();
        }
    }
}

// Work-counter slots (16 u32 apart) handed out round robin, so concurrent
// traces on different streams do not share a counter.
static std::atomic<uint32_t> g_slot{0};
// Resident blocks per SM: [closest] for the per-lane kernel, [2 + closest]
// for the cooperative one, [4 + closest] for its small-wavefront form; [6 + 2
// record] for the any-hit kernel, [7 + 2 record] for its small-wavefront form.
static int g_blocks_per_sm[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
static int g_num_sms = 0;
static uint32_t g_refill = 6;  // 4 to 8 within 1 % on bounce-1 rays, 6 the best sum

void set_trace_refill(uint32_t refill) { g_refill = refill < 1 ? 1 : (refill > 32 ? 32 : refill); }
static uint32_t g_postpone = 0;
void set_trace_postpone(uint32_t lanes) { g_postpone = lanes > 32 ? 32 : lanes; }
// Cooperative-test batch and node steps per loop iteration, [0] for any-hit
// rays, [1] for closest-hit rays.  The kernel takes twice the steps, since a
// lane goes on past its first triangles (any hit two more: its iterations
// end early by themselves), and tests once half the batch is pending.  So
// any-hit rays test after every iteration of up to eight node steps (a ray
// stops at its first hit: deferring tests only adds node steps, 1-3 % slower
// from batch 8 on), closest-hit rays at 12 pairs over iterations of four
// (3, 5, 6 and 8 steps: 1.5, 0.5, 1 and 5 % slower on the courtyard's sorted
// bounce-1 rays; 16 pairs equal there, 1 % slower on the city's and 4 % on a
// 57K-ray wavefront).
static uint32_t g_batch[2] = {1, 24};
static uint32_t g_steps[2] = {3, 2};
static uint32_t kernel_batch(bool closest) { return (g_batch[closest ? 1 : 0] + 1) / 2; }
// lanes: rays that the grid holds at once.  A wavefront that fits has no
// refills, so its any-hit iterations don't end early: four steps (57K soup
// rays: 109 us, 114 with eight).
static uint32_t kernel_steps(bool closest, uint32_t n, uint32_t lanes) {
    if (closest) return 2 * g_steps[1];
    const uint32_t steps = 2 * g_steps[0] + 2;
    return n <= lanes && steps > 4 ? 4 : steps;
}
void set_trace_steps(uint32_t steps, bool closest) {
    g_steps[closest ? 1 : 0] = steps < 1 ? 1 : (steps > 8 ? 8 : steps);
}
uint32_t get_trace_steps(bool closest) { return g_steps[closest ? 1 : 0]; }
void set_trace_batch(uint32_t pairs, bool closest) {
    g_batch[closest ? 1 : 0] = pairs < 1 ? 1 : (pairs > 32 ? 32 : pairs);
}
uint32_t get_trace_batch(bool closest) { return g_batch[closest ? 1 : 0]; }
static bool g_coop = true;
void set_trace_coop(bool on) { g_coop = on; }
bool get_trace_coop() { return g_coop; }
uint32_t get_trace_refill() { return g_refill; }
static bool g_count = false;
void set_trace_count(bool on) { g_count = on; }
bool get_trace_count() { return g_count; }

// SM count and resident blocks of the persistent kernel (host queries that
// must not run inside a stream capture; the renderer calls this first).
cudaError_t trace_prepare() {
    if (g_num_sms != 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_per_sm[0], k_trace_bvh8<false, false>, kBlock, 0);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_per_sm[1], k_trace_bvh8<true, false>, kBlock, 0);
    const void* coop[8] = {(const void*)k_trace_bvh8_coop<false, false, 4>, (const void*)k_trace_bvh8_coop<true, false, 4>,
                           (const void*)k_trace_bvh8_coop<false, false, 3>, (const void*)k_trace_bvh8_coop<true, false, 3>,
                           (const void*)k_any_bvh8<false, 4>, (const void*)k_any_bvh8<false, 3>,
                           (const void*)k_any_bvh8<true, 4>, (const void*)k_any_bvh8<true, 3>};
    for (int k = 0; k < 8 && e == cudaSuccess; ++k)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_per_sm[2 + k], coop[k], kBlock, 0);
    if (e == cudaSuccess) g_num_sms = sms;
    return e;
}

cudaError_t trace_counters(uint64_t out[4], bool reset) {
    unsigned long long v[4];
    cudaError_t e = cudaMemcpyFromSymbol(v, g_counts, sizeof(v));
    if (e != cudaSuccess) return e;
    for (int i = 0; i < 4; ++i) out[i] = v[i];
    if (reset) {
        unsigned long long z[4] = {0, 0, 0, 0};
        e = cudaMemcpyToSymbol(g_counts, z, sizeof(z));
    }
    return e;
}
uint32_t get_trace_postpone() { return g_postpone; }

cudaError_t launch_trace(const SceneDevice& sc, int kind, const wfpt_ray* rays, wfpt_hit* results,
                         const uint32_t* ray_index, uint32_t n, const uint32_t* n_dev, int closest,
                         cudaStream_t s, uint32_t* own_work, bool shared) {
    if (n == 0) return cudaSuccess;
    // A scene built without this BVH kind has no buffers for it.
    if (kind == WFPT_BVH8_Q8 ? (!sc.bvh8_nodes || !sc.bvh8_tris) : (!sc.bvh2_nodes || !sc.bvh2_tris))
        return cudaErrorInvalidValue;
    unsigned grid = (n + kBlock - 1) / kBlock;
    const float4* rr = reinterpret_cast<const float4*>(rays);
    int4* out = reinterpret_cast<int4*>(results);
    if (kind == WFPT_BVH8_Q8) {
        if (g_num_sms == 0) {
            cudaError_t e = trace_prepare();
            if (e != cudaSuccess) return e;
        }
        // The cooperative kernel packs a triangle record into 27 bits.
        const bool coop = g_coop && sc.bvh8_num_tris < (1u << kRecBits);
        const bool small = coop && n < kCoopLargeMin && !shared;
        unsigned pgrid = (unsigned)(g_num_sms * g_blocks_per_sm[(coop ? (small ? 4 : 2) : 0) + (closest ? 1 : 0)]);
        if (pgrid == 0) pgrid = 1;
        const uint32_t lanes = pgrid * kBlock;
        if (grid < pgrid) pgrid = grid;
        uint32_t* work = own_work ? own_work : sc.work + 16 * (g_slot.fetch_add(1) % kWorkSlots);
        // Counted any-hit records come from the kernel with a ring at batch 1: the
        // same node steps and tests as without.
        if (coop && !closest && !g_count && kernel_batch(false) <= 1u) {
            const unsigned resident = std::max(1u, (unsigned)(g_num_sms * g_blocks_per_sm[small ? 9 : 8]));
            auto k8 = small ? k_any_bvh8<true, 3> : k_any_bvh8<true, 4>;
            k8<<<std::min((n + kBlock - 1) / kBlock, resident), kBlock, 0, s>>>(
                sc.bvh8_nodes, sc.bvh8_tris, rr, out, ray_index, n, n_dev, work, g_refill,
                kernel_steps(false, n, resident * kBlock));
        } else if (coop) {
            auto k8 = closest ? (g_count ? k_trace_bvh8_coop<true, true, 4> : k_trace_bvh8_coop<true, false, 4>)
                              : (g_count ? k_trace_bvh8_coop<false, true, 4> : k_trace_bvh8_coop<false, false, 4>);
            if (small) {
                k8 = closest ? (g_count ? k_trace_bvh8_coop<true, true, 3> : k_trace_bvh8_coop<true, false, 3>)
                             : (g_count ? k_trace_bvh8_coop<false, true, 3> : k_trace_bvh8_coop<false, false, 3>);
            }
            k8<<<pgrid, kBlock, 0, s>>>(sc.bvh8_nodes, sc.bvh8_tris, rr, out, ray_index, n, n_dev, work, g_refill,
                                        kernel_batch(closest != 0), kernel_steps(closest != 0, n, lanes));
        } else {
            auto k8 = closest ? (g_count ? k_trace_bvh8<true, true> : k_trace_bvh8<true, false>)
                              : (g_count ? k_trace_bvh8<false, true> : k_trace_bvh8<false, false>);
            k8<<<pgrid, kBlock, 0, s>>>(sc.bvh8_nodes, sc.bvh8_tris, rr, out, ray_index, n, n_dev, work, g_refill,
                                        g_postpone);
        }
    } else {
        if (own_work != nullptr && n_dev != nullptr && n >= kBvh2RefillMin) {
            auto k2 = closest ? (g_count ? k_trace_bvh2_persistent<true, true> : k_trace_bvh2_persistent<true, false>)
                              : (g_count ? k_trace_bvh2_persistent<false, true> : k_trace_bvh2_persistent<false, false>);
            k2<<<std::min(grid, kBvh2Grid), kBlock, 0, s>>>(sc.bvh2_nodes, sc.bvh2_tris, rr, out, ray_index, n, n_dev,
                                                            own_work);
        } else if (n >= kBvh2SmallMin) {
            constexpr int B = kBvh2SmallBlock, P = kBvh2SmallPerSm;
            auto k2 = closest ? (g_count ? k_trace_bvh2<true, true, B, P> : k_trace_bvh2<true, false, B, P>)
                              : (g_count ? k_trace_bvh2<false, true, B, P> : k_trace_bvh2<false, false, B, P>);
            k2<<<(n + B - 1) / B, B, 0, s>>>(sc.bvh2_nodes, sc.bvh2_tris, rr, out, ray_index, n, n_dev);
        } else {
            auto k2 = closest ? (g_count ? k_trace_bvh2<true, true, kBlock, 1> : k_trace_bvh2<true, false, kBlock, 1>)
                              : (g_count ? k_trace_bvh2<false, true, kBlock, 1> : k_trace_bvh2<false, false, kBlock, 1>);
            k2<<<grid, kBlock, 0, s>>>(sc.bvh2_nodes, sc.bvh2_tris, rr, out, ray_index, n, n_dev);
        }
    }
    count_launch();
    return cudaGetLastError();
}

bool occluded_ready(const SceneDevice& sc, int kind) {
    return kind != WFPT_BVH8_Q8 || (g_coop && sc.bvh8_num_tris < (1u << kRecBits));
}

cudaError_t launch_occluded(const SceneDevice& sc, int kind, const wfpt_ray* rays, int32_t* occluded,
                            const uint32_t* ray_index, uint32_t n, const uint32_t* n_dev, cudaStream_t s,
                            uint32_t* work, bool shared) {
    if (n == 0) return cudaSuccess;
    if (kind == WFPT_BVH8_Q8 ? (!sc.bvh8_nodes || !sc.bvh8_tris) : (!sc.bvh2_nodes || !sc.bvh2_tris))
        return cudaErrorInvalidValue;
    const unsigned grid = (n + kBlock - 1) / kBlock;
    const float4* rr = reinterpret_cast<const float4*>(rays);
    if (kind == WFPT_BVH8_Q8) {
        if (g_num_sms == 0) {
            cudaError_t e = trace_prepare();
            if (e != cudaSuccess) return e;
        }
        const bool small = n < kCoopLargeMin && !shared;
        const unsigned resident = std::max(1u, (unsigned)(g_num_sms * g_blocks_per_sm[small ? 7 : 6]));
        auto k8 = small ? (g_count ? k_any_bvh8<false, 3, true> : k_any_bvh8<false, 3>)
                        : (g_count ? k_any_bvh8<false, 4, true> : k_any_bvh8<false, 4>);
        k8<<<std::min(grid, resident), kBlock, 0, s>>>(sc.bvh8_nodes, sc.bvh8_tris, rr, occluded, ray_index, n, n_dev,
                                                       work, g_refill, kernel_steps(false, n, resident * kBlock));
    } else {
        int4* out = reinterpret_cast<int4*>(occluded);
        constexpr int B = kBvh2SmallBlock, P = kBvh2SmallPerSm;
        if (n >= kBvh2RefillMin) {
            auto k2 = g_count ? k_trace_bvh2_persistent<false, true, true> : k_trace_bvh2_persistent<false, false, true>;
            k2<<<std::min(grid, kBvh2Grid), kBlock, 0, s>>>(sc.bvh2_nodes, sc.bvh2_tris, rr, out, ray_index, n, n_dev,
                                                            work);
        } else if (n >= kBvh2SmallMin) {
            auto k2 = g_count ? k_trace_bvh2<false, true, B, P, true> : k_trace_bvh2<false, false, B, P, true>;
            k2<<<(n + B - 1) / B, B, 0, s>>>(sc.bvh2_nodes, sc.bvh2_tris, rr, out, ray_index, n, n_dev);
        } else {
            auto k2 = g_count ? k_trace_bvh2<false, true, kBlock, 1, true> : k_trace_bvh2<false, false, kBlock, 1, true>;
            k2<<<grid, kBlock, 0, s>>>(sc.bvh2_nodes, sc.bvh2_tris, rr, out, ray_index, n, n_dev);
        }
    }
    count_launch();
    return cudaGetLastError();
}

}  // namespace wfpt
