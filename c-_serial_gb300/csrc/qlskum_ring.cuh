// A cloud's edge lists brought into shared memory by bulk copies (the mixed
// gradient kernel, qlskum_mixed.cu).
#pragma once
#include "qlskum_internal.h"
#include "qlskum_dev.cuh"

namespace qlskum {
namespace mixed {

// ---------------------------------------------- edge lists by bulk copies
// A slice's edge list (32 points of the sliced-ELL arrays) is contiguous in
// every array, so one bulk copy per array brings kRingEdges edges of 32 points
// into a warp's shared memory without registers or load instructions.
// Persistent warps keep a ring of kRingChunks such chunks: while a warp works on
// one, the next is in flight from DRAM, across the ends of its slices, and the
// gathers of a chunk's neighbours are issued together instead of each behind
// the load of its index.  Five edges: the usual ten take two chunks, and the
// five gathers leave registers for 24 warps per SM.
// Measured per launch of the gradient (us; before: one thread per point loading
// two edges per trip; 3 or 4 chunks, and 3, 4, 6 or 10 edges per chunk, are
// equal or slower on 1.02 M points): 9,600 points 9.6 -> 8.6, 101,617 15.3 ->
// 10.2, 1,024,000 52.6 -> 40.2 (the same bits).  The inner step, which gathers
// twice the bytes and streams 20 instead of 12 per edge, gains nothing there
// (55.7 and 55.5: 275 MB with the write-back, 5 TB/s) and keeps its form.
constexpr int kRingEdges = 5, kRingChunks = 2;
// Most warps of a block, whose barriers have their place in static shared
// memory; a launch of larger blocks (block_size up to 1,024) takes blocks of this many.
constexpr int kRingWarps = 16;

// Tells the host that a bulk copy did not arrive (DevCloud::fault).
__device__ __forceinline__ void set_fault(const DevCloud &c)
{
    if (!c.fault) return;
    *static_cast<volatile int *>(c.fault) = 1;
    __threadfence_system();
}

template <int NA> struct EdgeRing {
    static constexpr int CE = kRingEdges, NS = kRingChunks;
    const char *src[NA];
    int bytes[NA];              // per edge and lane
    unsigned buf, bar;          // this warp's shared memory: NS chunks, NS barriers
    int stage = 0;
    unsigned phase = 0;
    // the next chunk to fetch: edges [pj, pj + CE) of slice ps (width pw, first edge pbase)
    int ps, pj = 0, pw = 0, nslices, step;
    long long pbase = 0;
    // the slice after it, loaded ahead
    int nb_ahead = 0;
    long long base_ahead = 0;

    __device__ __forceinline__ void look(const DevCloud &c, int s)
    {
        const int i = 32 * s + (threadIdx.x & 31);
        nb_ahead = s < nslices && i < c.n ? c.nbhs[i] : 0;
        base_ahead = s < nslices ? c.slice_base[s] : 0;
    }

    // Moves on to the next slice that has edges.
    __device__ __forceinline__ void advance(const DevCloud &c)
    {
        pj = 0;
        do {
            ps += step;
            pw = __reduce_max_sync(0xffffffffu, nb_ahead);
            pbase = base_ahead;
            if (ps < nslices) look(c, ps + step);
        } while (pw == 0 && ps < nslices);
    }

    __device__ __forceinline__ void fetch(const DevCloud &c, int st, unsigned long long pol)
    {
        if (ps >= nslices) return;
        if ((threadIdx.x & 31) == 0) {
            const int m = min(CE, pw - pj);
            unsigned per = 0, dst = buf + st * chunk();
#pragma unroll
            for (int a = 0; a < NA; a++) per += bytes[a];
            mbar_expect(bar + 8 * st, 32u * m * per);
#pragma unroll
            for (int a = 0; a < NA; a++) {
                bulk_load(dst, src[a] + (pbase + 32LL * pj) * bytes[a], 32u * m * bytes[a], bar + 8 * st, pol);
                dst += 32u * CE * bytes[a];
            }
        }
        pj += CE;
        if (pj >= pw) advance(c);
    }

    __device__ __forceinline__ unsigned chunk() const
    {
        unsigned per = 0;
#pragma unroll
        for (int a = 0; a < NA; a++) per += bytes[a];
        return 32u * CE * per;
    }

    __device__ __forceinline__ void start(const DevCloud &c, int first, int stride, unsigned long long pol)
    {
        nslices = (c.n + 31) >> 5;
        step = stride;
        ps = first - stride;
        look(c, first);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int st = 0; st < NS; st++) mbar_init(bar + 8 * st, 1);
        __syncwarp();
        advance(c);
#pragma unroll
        for (int st = 0; st < NS; st++) fetch(c, st, pol);
    }

    // False (and the cloud's fault word set) if the chunk does not arrive within
    // the bound of mbar_wait; the other chunk in flight is waited for as well,
    // and the caller returns.
    __device__ __forceinline__ bool wait(const DevCloud &c)
    {
        if (mbar_wait(bar + 8 * stage, phase)) return true;
        set_fault(c);
        static_assert(NS == 2, "the other chunk in flight is named by stage ^ 1");
        mbar_wait(bar + 8 * (stage ^ 1), stage ? phase ^ 1 : phase);
        return false;
    }

    // The chunk is used up: its place takes the next one.
    __device__ __forceinline__ void next(const DevCloud &c, unsigned long long pol)
    {
        __syncwarp();
        fetch(c, stage, pol);
        if (++stage == NS) {
            stage = 0;
            phase ^= 1;
        }
    }
};

}  // namespace mixed
}  // namespace qlskum
