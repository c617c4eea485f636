// window.cuh -- block locations for a producer warp that walks a column in
// order, ahead of time.
//
// A tile's size depends on its blocks' widths, so the next tile's first block
// is known only when a tile is formed; loading its index entries then costs
// the producer a trip to memory per tile (2 us with the memory pipes full,
// which bounded the kernels it feeds).  The warp therefore keeps the entries of
// three windows of 32 blocks in registers, the third one on its way: a tile's
// entries come from the first two by shuffles.
#pragma once

#include "stream.cuh"

namespace ms {
namespace {

template <unsigned C>
struct BlockWindow {
    uint64_t e[C][3];  // index entries of blocks base + 32 i + lane
    uint64_t base, end;

    __device__ __forceinline__ uint64_t entry(const StreamCol &c, uint64_t b) const {
        if (b >= end) return 0;
        if (c.index) return __ldg(c.index + b);
        return idx_pack(b * 64ull * c.fixed_bw, c.fixed_bw);
    }
    __device__ __forceinline__ void init(const StreamCol *const (&cols)[C], uint64_t b_lo, uint64_t b_hi, unsigned lane) {
        base = b_lo;
        end = b_hi;
#pragma unroll
        for (unsigned c = 0; c < C; c++)
#pragma unroll
            for (unsigned i = 0; i < 3; i++) e[c][i] = entry(*cols[c], base + 32 * i + lane);
    }
    // moves the windows to block b, at most 32 blocks on
    __device__ __forceinline__ void advance(const StreamCol *const (&cols)[C], uint64_t b, unsigned lane) {
        if (b < base + 32) return;
        base += 32;
#pragma unroll
        for (unsigned c = 0; c < C; c++) {
            e[c][0] = e[c][1];
            e[c][1] = e[c][2];
            e[c][2] = entry(*cols[c], base + 64 + lane);
        }
    }
    // block b + lane of column c (b within the first window)
    __device__ __forceinline__ void get(unsigned c, uint64_t b, unsigned lane, uint64_t &off, unsigned &bw) const {
        const unsigned i = unsigned(b - base) + lane;
        const uint64_t x = __shfl_sync(0xFFFFFFFFu, e[c][0], i & 31u), y = __shfl_sync(0xFFFFFFFFu, e[c][1], i & 31u);
        const uint64_t v = i < 32 ? x : y;
        off = idx_off(v);
        bw = idx_bw(v);
    }
};

}  // namespace
}  // namespace ms
