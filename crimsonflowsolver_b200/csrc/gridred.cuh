// Grid-wide barrier that carries reductions, for the persistent cooperative
// kernels (all blocks co-resident).
//
// A counter-based barrier followed by a reduction over per-block partial sums
// costs two trips through the L2: arrive / wait, then read the partials.
// Here every block publishes each of its partial sums as one 16-byte packet
// {value, epoch} and waits until the packets of all blocks carry the epoch,
// so the values arrive with the barrier itself.  Every block sums the packets
// in block order: the result is the same bits in every block and on every
// run.  Measured (768 threads per block; one sum, without and with the blocks'
// global writes ordered before it): 1.2 / 2.0 us on 20 blocks, 1.4 / 2.3 on
// 74, 2.6 / 3.9 on 148, where every block's polls of all packets meet in the
// L2.  cooperative_groups' grid.sync takes 1.2 us on any of them, and with the
// writes before it and the partials read and summed after it 2.2-2.3.
//
// Packets of two consecutive epochs live in alternating regions: a block can
// be at most one epoch ahead of the slowest one, which is still reading the
// previous region.  Epochs grow monotonically over the launches that share a
// packet buffer, so the buffer is cleared once, at its allocation.
//
// Every wait is bounded.  A block whose wait runs out reports it to its threads
// and waits for nothing more: they pass the barriers that are left in the
// kernel's loops and leave them, and the other blocks follow when their own
// waits run out.
#pragma once

#include "common.cuh"

namespace crimson {

constexpr int kGrMaxBlocks = 160;              // blocks of a grid that reduces this way
constexpr int kGrPolls = kGrMaxBlocks / 32;    // packets per lane and value
#ifndef CRIMSON_GR_WAIT_CLOCKS
#define CRIMSON_GR_WAIT_CLOCKS (1LL << 32)
#endif
constexpr long long kGrWaitClocks = CRIMSON_GR_WAIT_CLOCKS;  // SM clocks before a wait gives up (about two seconds)

__device__ __forceinline__ void gr_publish(ulonglong2* p, double v, unsigned long long epoch) {
    asm volatile(
        "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
        "l"(__double_as_longlong(v)), "l"(epoch)
        : "memory");
}

__device__ __forceinline__ ulonglong2 gr_load(const ulonglong2* p) {
    ulonglong2 r;
    asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
                 : "=l"(r.x), "=l"(r.y)
                 : "l"(p)
                 : "memory");
    return r;
}

// Lane's share of the packets of all blocks: bit j stands for block
// lane + 32 j.
__device__ __forceinline__ unsigned gr_all_blocks() {
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < kGrPolls; ++j)
        if ((int)(threadIdx.x & 31) + 32 * j < (int)gridDim.x) m |= 1u << j;
    return m;
}

// Sum over a warp of the packets of the blocks in pend (per lane, as
// gr_all_blocks), every lane receiving it; waits until all of them carry the
// epoch or the limit since t0 (0: the first poll) has passed.
__device__ __forceinline__ double gr_collect(const ulonglong2* pk, unsigned pend, unsigned long long epoch, bool* fail,
                                             long long t0) {
    const int lane = threadIdx.x & 31;
    double v[kGrPolls];
#pragma unroll
    for (int j = 0; j < kGrPolls; ++j) v[j] = 0.0;
    while (__any_sync(0xffffffffu, pend)) {
        ulonglong2 r[kGrPolls];
#pragma unroll
        for (int j = 0; j < kGrPolls; ++j)
            if ((pend >> j) & 1) r[j] = gr_load(pk + lane + 32 * j);
#pragma unroll
        for (int j = 0; j < kGrPolls; ++j)
            if (((pend >> j) & 1) && r[j].y == epoch) {
                v[j] = __longlong_as_double((long long)r[j].x);
                pend &= ~(1u << j);
            }
        if (t0 == 0) t0 = clock64();
        if (__any_sync(0xffffffffu, clock64() - t0 > kGrWaitClocks)) {
            *fail = true;
            break;
        }
    }
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < kGrPolls; ++j) s += v[j];
    return warp_sum(s);
}

// Orders the block's global writes (made before a __syncthreads) ahead of
// the packets this thread publishes afterwards.
__device__ __forceinline__ void gr_release() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// After gr_collect: the collected blocks' writes are visible to this thread
// and, past a __syncthreads, to its block.
__device__ __forceinline__ void gr_acquire() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// The reductions of one barrier.  red[32 k + w]: warp w's partial of value k
// (shared memory); tot[k] (shared) receives the sums, valid on return for
// every thread.  Value 0 comes from every block and is the barrier itself;
// values 1 + 2 f and 2 + 2 f (f < nface) come only from the blocks whose
// own_faces has bit f -- the others' are zero -- and fpend[32 f + lane] says
// which these are (as gr_all_blocks).  Three values from every block take no
// longer than one (2.5 us on 148 blocks).  pk: two regions of kvals
// packets per block.  data: the block's global writes before the call are
// visible to all blocks after it.  Returns whether a thread of the block gave
// up a wait, in this call or before it (failed).
static __device__ __noinline__ bool grid_reduce(ulonglong2* pk, int kvals, const double* red, int nface,
                                                unsigned own_faces, const unsigned char* fpend, unsigned long long ep,
                                                bool data, double* tot, bool failed) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5, nv = 1 + 2 * nface;
    pk += (size_t)(ep & 1) * kvals * gridDim.x;
    bool fail = failed;
    // after a wait that ran out: one poll
    const long long t0 = failed ? -(1LL << 62) : 0;
    __syncthreads();
    for (int k = wid; k < nv; k += nw)
        if (k == 0 || ((own_faces >> ((k - 1) / 2)) & 1)) {
            const double v = warp_sum(lane < nw ? red[32 * k + lane] : 0.0);
            if (lane == 0) {
                if (data) gr_release();
                gr_publish(pk + (size_t)k * gridDim.x + blockIdx.x, v, ep);
            }
        }
    for (int k = wid; k < nv; k += nw) {
        const unsigned pend = k == 0 ? gr_all_blocks() : fpend[32 * ((k - 1) / 2) + lane];
        const double v = gr_collect(pk + (size_t)k * gridDim.x, pend, ep, &fail, t0);
        if (data) gr_acquire();
        if (lane == 0) tot[k] = v;
    }
    return __syncthreads_or(fail) != 0;
}

}  // namespace crimson
