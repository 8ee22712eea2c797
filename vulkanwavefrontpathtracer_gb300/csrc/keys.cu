// Morton key generation and the ray-reorder gather.
//
// Both are HBM-bound streaming kernels: Morton reads one 32-byte ray and
// writes a key (4 or 8 B) plus an index (4 B); reorder gathers one 32-byte
// ray and one slot-map entry by the sorted permutation, writes them in
// order and scatters the inverse slot map.
#include "common.cuh"
#include "morton.cuh"
#include "stages.cuh"

namespace wfpt {

template <int KIND>
__global__ void k_morton(const float4* __restrict__ rays, uint32_t n, const uint32_t* __restrict__ n_dev,
                         Box6 box, void* __restrict__ keys, uint32_t* __restrict__ indices) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= load_count(n, n_dev)) return;
    float4 r0 = rays[2 * i + 0];
    float4 r1 = rays[2 * i + 1];
    write_morton_key<KIND>(keys, i, r0, r1, box);
    indices[i] = i;
}

// Gathers beyond L2 (STREAM): the index, the gathered records and the
// written records are touched once, so they are loaded and stored with an
// L2 evict-first policy, and the L2 keeps the randomly accessed 4-byte slot
// map entries (each 32-byte sector of them is touched eight times, at random
// moments) for longer.  Random-permutation gathers of 32- / 48-byte records:
// 7 / 10 % faster at 2^22 rays, 26 / 20 % at 2^23 (beyond kSplitRecords the
// maps go apart); an evict-last policy on the slot maps instead was 3-12 %
// slower.
// Smaller gathers (a frame's 2.07M-ray wavefront, whose records the next
// kernel reads back from L2) keep plain accesses: the policy made 2^21 rays
// 5-10 % slower.
constexpr uint32_t kStreamRecords = 1u << 22;

__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
template <bool STREAM>
__device__ __forceinline__ uint4 load_record(const uint4* p, uint64_t pol) {
    if (!STREAM) return __ldg(p);
    uint4 v;
    asm volatile("ld.global.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p), "l"(pol));
    return v;
}
template <bool STREAM>
__device__ __forceinline__ void store_record(uint4* p, uint4 v, uint64_t pol) {
    if (!STREAM) {
        *p = v;
        return;
    }
    asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w), "l"(pol)
                 : "memory");
}

// reorderRays.comp:37-45.  out_i2s (nullable, here and below): a renderer's path
// rays are never looked up by index (2.07M rays 39 -> 31 us without).
template <bool STREAM>
__global__ void k_reorder(const uint32_t* __restrict__ idx, const uint4* __restrict__ in_rays,
                          uint4* __restrict__ out_rays, const int32_t* __restrict__ in_s2i,
                          int32_t* __restrict__ out_s2i, int32_t* __restrict__ out_i2s, uint32_t n,
                          const uint32_t* __restrict__ n_dev, bool wide) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= load_count(n, n_dev)) return;
    const uint64_t pol = STREAM ? l2_evict_first_policy() : 0u;
    uint32_t old = STREAM ? __ldcs(idx + i) : idx[i];
    int32_t index = in_s2i[old];
    if (!STREAM && wide) {
        float4 a, b;
        load32(reinterpret_cast<const float4*>(in_rays) + 2 * (size_t)old, a, b);
        store_ray(reinterpret_cast<float4*>(out_rays), i, a, b, true);
    } else {
        uint4 a = load_record<STREAM>(in_rays + 2 * (size_t)old + 0, pol);
        uint4 b = load_record<STREAM>(in_rays + 2 * (size_t)old + 1, pol);
        store_record<STREAM>(out_rays + 2 * (size_t)i + 0, a, pol);
        store_record<STREAM>(out_rays + 2 * (size_t)i + 1, b, pol);
    }
    if (STREAM) {
        __stcs(out_s2i + i, index);
    } else {
        out_s2i[i] = index;
    }
    if (out_i2s != nullptr) out_i2s[index] = (int32_t)i;
}

// The same gather for records of C x 16 bytes (ray records with a payload,
// 48 B = 3 chunks).  One thread per record: the C 16-byte loads of a record
// are issued together; stores are coalesced across the warp.  The slot maps
// are optional (in_s2i == nullptr: plain gather).
template <int C, bool STREAM>
__global__ void k_reorder_records(const uint32_t* __restrict__ idx, const uint4* __restrict__ in_rec,
                                  uint4* __restrict__ out_rec, const int32_t* __restrict__ in_s2i,
                                  int32_t* __restrict__ out_s2i, int32_t* __restrict__ out_i2s, uint32_t n,
                                  const uint32_t* __restrict__ n_dev) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= load_count(n, n_dev)) return;
    const uint64_t pol = STREAM ? l2_evict_first_policy() : 0u;
    uint32_t old = STREAM ? __ldcs(idx + i) : idx[i];
    uint4 v[C];
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = load_record<STREAM>(in_rec + (size_t)C * old + c, pol);
#pragma unroll
    for (int c = 0; c < C; ++c) store_record<STREAM>(out_rec + (size_t)C * i + c, v[c], pol);
    int32_t index = in_s2i[old];
    if (STREAM) {
        __stcs(out_s2i + i, index);
    } else {
        out_s2i[i] = index;
    }
    out_i2s[index] = (int32_t)i;
}

// The gather of wavefronts far beyond L2, in three launches, and of records
// without slot maps at any size.  A fused gather touches three random
// streams at once (the records, the old slot map's entries and the inverse
// map's entries), so from about 10M records on none of them stays in L2 and
// every 4-byte map access moves a DRAM sector of its own.  Apart, each map's
// table is what L2 holds while it is accessed.  Random permutations,
// fused / split: 0.92 / 0.55 ms at 2^24 32-byte records (1.09 / 0.66 ms at
// 48 bytes), 2.33 / 1.25 ms at 2^25; equal at 2^23 and slower below (the map
// passes' launches, about 4 us each, and their second reads).
constexpr uint32_t kSplitRecords = 10u << 20;
// Map entries per range pass.  A map of more entries than this (64 MB) is
// gathered or scattered in ranges, one launch a range, each over all n
// indexes (streamed) but touching only the map entries of its range, which
// then stay in L2: scatter 0.53 -> 0.21 ms, gather 0.31 -> 0.23 ms at 2^25
// (two ranges), 2.06 -> 0.60 and 1.00 -> 0.67 ms at 2^26 (four).  More ranges
// than needed cost another pass over the indexes each (2^24: 0.08 -> 0.09 ms).
constexpr uint32_t kMapRange = 1u << 24;

// Records by permutation: one lane per 16-byte chunk, so a warp's loads take
// each record's chunks in one request and its stores are whole lines; four
// chunks in flight per lane.  Bound by DRAM's random 32- to 64-byte reads
// (48-byte records, 2^24: 0.51 ms = 3.3 TB/s algorithmic; a lane per record
// took 0.56 ms, 1.24 against 1.03 ms at 2^25).
constexpr int kGatherUnroll = 4;
template <int C>
__global__ void __launch_bounds__(kBlock) k_gather_chunks(const uint32_t* __restrict__ idx,
                                                          const uint4* __restrict__ in_rec,
                                                          uint4* __restrict__ out_rec, uint32_t n,
                                                          const uint32_t* __restrict__ n_dev) {
    const size_t total = (size_t)load_count(n, n_dev) * C;
    const size_t t0 = (size_t)blockIdx.x * (kBlock * kGatherUnroll) + threadIdx.x;
    uint4 v[kGatherUnroll];
#pragma unroll
    for (int u = 0; u < kGatherUnroll; ++u) {
        const size_t t = t0 + u * kBlock;
        if (t < total) {
            // total <= 4 (2^30 - 1): a chunk number below it fits 32 bits.
            const uint32_t i = (uint32_t)t / C, c = (uint32_t)t - i * C;
            v[u] = __ldg(in_rec + (size_t)C * __ldg(idx + i) + c);
        }
    }
#pragma unroll
    for (int u = 0; u < kGatherUnroll; ++u) {
        const size_t t = t0 + u * kBlock;
        if (t < total) __stcs(out_rec + t, v[u]);
    }
}

// Four consecutive entries of a 4-byte array, streamed: one 16-byte access
// when the array allows it (VEC: its address is a multiple of 16).
template <bool VEC>
__device__ __forceinline__ uint4 load4(const uint32_t* p) {
    if (VEC) return __ldcs(reinterpret_cast<const uint4*>(p));
    return make_uint4(__ldcs(p), __ldcs(p + 1), __ldcs(p + 2), __ldcs(p + 3));
}

// out_s2i[i] = in_s2i[idx[i]] for the idx[i] in [lo, lo + len).
template <bool VEC>
__global__ void __launch_bounds__(kBlock) k_map_gather(const uint32_t* __restrict__ idx,
                                                       const int32_t* __restrict__ in_s2i,
                                                       int32_t* __restrict__ out_s2i, uint32_t n,
                                                       const uint32_t* __restrict__ n_dev, uint32_t lo,
                                                       uint32_t len) {
    const uint32_t count = load_count(n, n_dev);
    const uint32_t i = (blockIdx.x * kBlock + threadIdx.x) * 4u;
    if (i + 3u < count) {
        const uint4 q = load4<VEC>(idx + i);
        const bool in[4] = {q.x - lo < len, q.y - lo < len, q.z - lo < len, q.w - lo < len};
        int4 v = make_int4(0, 0, 0, 0);
        if (in[0]) v.x = in_s2i[q.x];
        if (in[1]) v.y = in_s2i[q.y];
        if (in[2]) v.z = in_s2i[q.z];
        if (in[3]) v.w = in_s2i[q.w];
        if (VEC && in[0] && in[1] && in[2] && in[3]) {
            __stcs(reinterpret_cast<int4*>(out_s2i + i), v);
        } else {
            if (in[0]) out_s2i[i] = v.x;
            if (in[1]) out_s2i[i + 1] = v.y;
            if (in[2]) out_s2i[i + 2] = v.z;
            if (in[3]) out_s2i[i + 3] = v.w;
        }
    } else {
        for (uint32_t j = i; j < count; ++j) {
            const uint32_t q = idx[j];
            if (q - lo < len) out_s2i[j] = in_s2i[q];
        }
    }
}

// out_i2s[out_s2i[i]] = i for the out_s2i[i] in [lo, lo + len).
template <bool VEC>
__global__ void __launch_bounds__(kBlock) k_map_scatter(const int32_t* __restrict__ out_s2i,
                                                        int32_t* __restrict__ out_i2s, uint32_t n,
                                                        const uint32_t* __restrict__ n_dev, uint32_t lo,
                                                        uint32_t len) {
    const uint32_t count = load_count(n, n_dev);
    const uint32_t i = (blockIdx.x * kBlock + threadIdx.x) * 4u;
    if (i + 3u < count) {
        const uint4 q = load4<VEC>(reinterpret_cast<const uint32_t*>(out_s2i + i));
        if (q.x - lo < len) out_i2s[(int32_t)q.x] = (int32_t)i;
        if (q.y - lo < len) out_i2s[(int32_t)q.y] = (int32_t)i + 1;
        if (q.z - lo < len) out_i2s[(int32_t)q.z] = (int32_t)i + 2;
        if (q.w - lo < len) out_i2s[(int32_t)q.w] = (int32_t)i + 3;
    } else {
        for (uint32_t j = i; j < count; ++j) {
            const uint32_t q = (uint32_t)out_s2i[j];
            if (q - lo < len) out_i2s[(int32_t)q] = (int32_t)j;
        }
    }
}

template <int C>
static cudaError_t launch_gather(const uint32_t* idx, const uint4* in, uint4* out, uint32_t n, const uint32_t* n_dev,
                                 cudaStream_t s) {
    const size_t per_block = (size_t)kBlock * kGatherUnroll;
    const unsigned grid = (unsigned)(((size_t)n * C + per_block - 1) / per_block);
    k_gather_chunks<C><<<grid, kBlock, 0, s>>>(idx, in, out, n, n_dev);
    count_launch();
    return cudaGetLastError();
}

// Both slot maps, range by range.  The old map is indexed by ray (below n);
// its values are whatever the caller numbers rays by (pixels in a renderer),
// so the last scatter range takes every value past it too.
static cudaError_t launch_maps(const uint32_t* idx, const int32_t* in_s2i, int32_t* out_s2i, int32_t* out_i2s,
                               uint32_t n, const uint32_t* n_dev, cudaStream_t s) {
    const unsigned grid = (unsigned)(((size_t)n + 4 * kBlock - 1) / (4 * kBlock));
    const uint32_t ranges = (n + kMapRange - 1) / kMapRange;
    const uint32_t step = (n + ranges - 1) / ranges;
    const bool vec = ((reinterpret_cast<uintptr_t>(idx) | reinterpret_cast<uintptr_t>(out_s2i)) & 15u) == 0;
    auto gather = vec ? k_map_gather<true> : k_map_gather<false>;
    auto scatter = vec ? k_map_scatter<true> : k_map_scatter<false>;
    // In place over the index array (a thread reads its entries before it writes
    // them) it is one range: a second one would read the first one's output.
    const uint32_t gathers = reinterpret_cast<const void*>(idx) == out_s2i ? 1u : ranges;
    for (uint32_t r = 0; r < gathers; ++r) {
        const uint32_t lo = r * step;
        gather<<<grid, kBlock, 0, s>>>(idx, in_s2i, out_s2i, n, n_dev, lo, r + 1 == gathers ? 0xFFFFFFFFu - lo : step);
    }
    for (uint32_t r = 0; r < ranges && out_i2s != nullptr; ++r) {
        const uint32_t lo = r * step;
        scatter<<<grid, kBlock, 0, s>>>(out_s2i, out_i2s, n, n_dev, lo, r + 1 == ranges ? 0xFFFFFFFFu - lo : step);
    }
    count_launch(out_i2s != nullptr ? gathers + ranges : gathers);
    return cudaGetLastError();
}

cudaError_t launch_morton(const wfpt_ray* rays, uint32_t n, const uint32_t* n_dev, const float* smin,
                          const float* ssize, int kind, void* keys, uint32_t* indices, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    Box6 box;
    for (int k = 0; k < 3; ++k) {
        box.smin[k] = smin[k];
        box.ssize[k] = ssize[k];
    }
    unsigned grid = (n + kBlock - 1) / kBlock;
    const float4* r = reinterpret_cast<const float4*>(rays);
    switch (kind) {
        case WFPT_MORTON_AILA32: k_morton<WFPT_MORTON_AILA32><<<grid, kBlock, 0, s>>>(r, n, n_dev, box, keys, indices); break;
        case WFPT_MORTON_6D48: k_morton<WFPT_MORTON_6D48><<<grid, kBlock, 0, s>>>(r, n, n_dev, box, keys, indices); break;
        default: k_morton<WFPT_MORTON_6D64><<<grid, kBlock, 0, s>>>(r, n, n_dev, box, keys, indices); break;
    }
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_reorder(const uint32_t* idx, const wfpt_ray* in_rays, wfpt_ray* out_rays,
                           const int32_t* in_s2i, int32_t* out_s2i, int32_t* out_i2s, uint32_t n,
                           const uint32_t* n_dev, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (n >= kSplitRecords) {
        cudaError_t e = launch_gather<2>(idx, reinterpret_cast<const uint4*>(in_rays),
                                         reinterpret_cast<uint4*>(out_rays), n, n_dev, s);
        return e != cudaSuccess ? e : launch_maps(idx, in_s2i, out_s2i, out_i2s, n, n_dev, s);
    }
    unsigned grid = (n + kBlock - 1) / kBlock;
    auto k = n >= kStreamRecords ? k_reorder<true> : k_reorder<false>;
    k<<<grid, kBlock, 0, s>>>(idx, reinterpret_cast<const uint4*>(in_rays), reinterpret_cast<uint4*>(out_rays), in_s2i,
                              out_s2i, out_i2s, n, n_dev, wide_rays(in_rays) && wide_rays(out_rays));
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_reorder_records(const uint32_t* idx, const void* in_records, void* out_records,
                                   uint32_t record_bytes, const int32_t* in_s2i, int32_t* out_s2i, int32_t* out_i2s,
                                   uint32_t n, const uint32_t* n_dev, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    unsigned grid = (n + kBlock - 1) / kBlock;
    const uint4* in = static_cast<const uint4*>(in_records);
    uint4* out = static_cast<uint4*>(out_records);
    if (n >= kSplitRecords || in_s2i == nullptr) {
        cudaError_t e = cudaErrorInvalidValue;
        switch (record_bytes) {
            case 16: e = launch_gather<1>(idx, in, out, n, n_dev, s); break;
            case 32: e = launch_gather<2>(idx, in, out, n, n_dev, s); break;
            case 48: e = launch_gather<3>(idx, in, out, n, n_dev, s); break;
            case 64: e = launch_gather<4>(idx, in, out, n, n_dev, s); break;
            default: break;
        }
        if (e != cudaSuccess || in_s2i == nullptr) return e;
        return launch_maps(idx, in_s2i, out_s2i, out_i2s, n, n_dev, s);
    }
    const bool st = n >= kStreamRecords;
    switch (record_bytes) {
#define WFPT_REORDER_REC(B, C)                                                                                       \
    case B:                                                                                                          \
        (st ? k_reorder_records<C, true> : k_reorder_records<C, false>)<<<grid, kBlock, 0, s>>>(                     \
            idx, in, out, in_s2i, out_s2i, out_i2s, n, n_dev);                                                       \
        break;
        WFPT_REORDER_REC(16, 1) WFPT_REORDER_REC(32, 2) WFPT_REORDER_REC(48, 3) WFPT_REORDER_REC(64, 4)
#undef WFPT_REORDER_REC
        default: return cudaErrorInvalidValue;
    }
    count_launch();
    return cudaGetLastError();
}

}  // namespace wfpt
