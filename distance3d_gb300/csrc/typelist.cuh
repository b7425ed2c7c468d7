// typelist.cuh -- a block's tasks listed by kind, so that its warps take
// chunks of one kind.  The lanes of a warp then run the same FP64 support on
// different colliders; an FP64 instruction costs the pipe the same however few
// lanes are active.
//
//   every thread   pos = atomicAdd(cnt + bin, count)      (cnt cleared before)
//   __syncthreads
//   every warp     Chunks c = chunks_of(cnt, bins, size)  (size: tasks per chunk of bin = lane)
//   every thread   list[c.start(bin) + pos ...] = task
//   __syncthreads
//   every warp     while (c.take(&next, bin, first, count)) ...
#pragma once

#include <cuda_runtime.h>

#include "d3d_device.cuh"

namespace d3d {

// Lane b holds bin b's task count, its end and its chunks' end in the list.
struct Chunks {
    int size, count, end, chunk_count, chunk_end, total;

    // first list position of a bin (every lane calls, each with its own bin)
    __device__ __forceinline__ int start(int bin) const { return __shfl_sync(0xffffffffu, end - count, bin); }

    // The warp's next chunk (later bins first): its bin and its tasks' first list position and number.
    __device__ __forceinline__ bool take(int* next, int& bin, int& first, int& n) const {
        constexpr unsigned all = 0xffffffffu;
        int x = 0;
        if ((threadIdx.x & 31) == 0) x = atomicAdd(next, 1);
        x = total - 1 - __shfl_sync(all, x, 0);
        if (x < 0) return false;
        bin = __popc(__ballot_sync(all, chunk_end <= x));
        const int s = __shfl_sync(all, size, bin);
        const int k = (x - __shfl_sync(all, chunk_end - chunk_count, bin)) * s;
        first = __shfl_sync(all, end - count, bin) + k;
        n = min(s, __shfl_sync(all, count, bin) - k);
        return true;
    }
};

__device__ __forceinline__ Chunks chunks_of(const int* cnt, int bins, int size) {
    constexpr unsigned all = 0xffffffffu;
    const int ln = threadIdx.x & 31;
    Chunks c;
    c.size = size;
    c.count = ln < bins ? cnt[ln] : 0;
    c.chunk_count = (c.count + size - 1) / size;
    c.end = c.count;
    c.chunk_end = c.chunk_count;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const int a = __shfl_up_sync(all, c.end, k), b = __shfl_up_sync(all, c.chunk_end, k);
        if (ln >= k) {
            c.end += a;
            c.chunk_end += b;
        }
    }
    c.total = __shfl_sync(all, c.chunk_end, 31);
    return c;
}

// Bins of the support tasks: a collider's type without and with a margin, then
// the hulls whose vertex is not known and has to be searched.
constexpr int kSupportTypes = 10;
constexpr int kSearchBin = 2 * kSupportTypes;
constexpr int kSupportBins = kSearchBin + 1;
__device__ __forceinline__ int support_bin(int type, int wrapped) {
    return 2 * min(max(type, 0), kSupportTypes - 1) + (wrapped ? 1 : 0);
}

// hull_argmax in FP32 with the lanes of the whole warp on one hull: the first
// maximum of V . d (-0 equal to +0, a NaN at vertex 0 kept, later NaNs
// skipped).  Every lane calls it with the same arguments and gets the index.
__device__ __forceinline__ int warp_hull_argmax(const float* verts, int off, int nv, V3<float> d) {
    constexpr unsigned all = 0xffffffffu;
    if (nv == 1) return 0;
    unsigned best = 0u;
    int bi = 0x7fffffff;
    bool nan0 = false;
    for (int k = threadIdx.x & 31; k < nv; k += 32) {
        const V3<float> v = load_vertex(verts, off + k);
        const float x = dot102(v.x, v.y, v.z, d.x, d.y, d.z);
        const unsigned u = x == 0.f ? 0u : __float_as_uint(x);
        const unsigned key = x != x ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
        if (k == 0 && key == 0u) nan0 = true;
        if (key > best) {
            best = key;
            bi = k;
        }
    }
    const unsigned m = __reduce_max_sync(all, best);
    const unsigned i = __reduce_min_sync(all, best == m ? (unsigned)bi : 0xffffffffu);
    return (__any_sync(all, nan0) || i >= (unsigned)nv) ? 0 : (int)i;
}

}  // namespace d3d
