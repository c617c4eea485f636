// rounds.cuh -- one pass over a column whose output offsets depend on
// everything before them (block widths, run counts).
//
// Persistent CTAs, one per SM, take tiles of 6144 rows in rounds: tile
// r * gridDim + c is CTA c's in round r.  Stages overlap: bulk copies into
// shared-memory buffers; the first half of the warps takes tile r into
// registers, publishes one word about it and prepares its output in place; the
// other half asks for the words of round r - 1 and writes out tile r - 2, whose
// place it gets from the words of its round, requested a round ago, and from
// the sum over the rounds before; then the buffer takes tile r + 2.  Four
// buffers of 48 KB: one being analysed, two waiting for their words, one being
// filled.
//
// What this is built around: with the memory pipes full a read of a published
// word takes more than a microsecond, most of a round, so no stage may wait
// for one; a look-back by CTAs that load, analyse, look back and write one
// after another took 12 us per tile.  2^27 rows of 20 bits (dynamic_vbp):
// 265 us, of which reading the rows and writing the blocks take 215 at the
// copy rate; with an analysis pass, a scan and a packing pass over the rows
// again 395 us.
//
// The CTAs wait on one another, so the kernel is launched cooperatively
// (all CTAs resident or an error).  Every wait is bounded; a wait that gives
// up sets `fail`, after which no further wait is made, but every thread goes
// through the same barriers to the end, so that none is left at one.
#pragma once

#include "tma.cuh"

namespace ms {
namespace {

constexpr unsigned kRdWarps = 6, kRdHalf = 32 * kRdWarps, kRdThreads = 2 * kRdHalf;
constexpr unsigned kRdRows = 1024 * kRdWarps;  // rows per tile
constexpr unsigned kRdBufs = 4;
// A tile in shared memory starts at byte 128 of its buffer; up to 8 rows before
// it end there.
constexpr unsigned kRdHead = 128, kRdBuf = kRdHead + 8 * kRdRows, kRdSmem = kRdBufs * kRdBuf;

__device__ __forceinline__ unsigned rd_row(unsigned r) { return kRdHead + 8u * r; }
__device__ __forceinline__ uint8_t *rd_buf(uint8_t *smem, unsigned r) { return smem + r % kRdBufs * kRdBuf; }
// barrier of one half of the warps
__device__ __forceinline__ void rd_bar(unsigned half) {
    asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "r"(kRdHalf) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

struct RdShared {
    uint64_t full[kRdBufs];
    unsigned lower[kRdWarps], total[kRdWarps], lower_last[kRdWarps], total_last[kRdWarps];
    volatile unsigned fail;
};

__device__ __forceinline__ void rd_init(RdShared &sh) {
    if (threadIdx.x == 0) {
        for (unsigned i = 0; i < kRdBufs; i++) mbar_init(sh.full + i, 1);
        mbar_fence_init();
        sh.fail = 0;
    }
    __syncthreads();
}

// waits for the copy of the CTA's tile of round r
__device__ __forceinline__ void rd_full(RdShared &sh, unsigned r) {
    if (!mbar_wait(sh.full + r % kRdBufs, (r / kRdBufs) & 1u)) sh.fail = 1;
}

// Bulk copy of the rows [row0, row0 + rows) and `before` rows in front of
// them (0, 2 or 8) into `buf`, by one thread (one copy: issuing one takes some
// 60 cycles).  An odd last row, which a 16-byte copy cannot end on, is left
// to the caller.
__device__ __forceinline__ void rd_load(uint8_t *buf, uint64_t *full, const uint64_t *in, uint64_t row0, unsigned rows,
                                        unsigned before) {
    const unsigned bytes = 8u * ((rows & ~1u) + before);
    mbar_arrive_expect_tx(full, bytes);
    if (bytes) bulk_g2s(buf + kRdHead - 8u * before, in + row0 - before, bytes, full);
}

// Published words, one per tile, each in a line of its own (neighbours in one
// line made a word some 5 us late: the line is written by many SMs while
// others read it): bit 0 set, above it 13 bits that are summed up (block
// widths, runs) and 13 bits of which the latest counts (last run head + 1, 0
// for none).  kStride: words from one tile's to the next.
constexpr unsigned kRdWordStride = 32;
template <unsigned kStride = kRdWordStride>
__device__ __forceinline__ void rd_publish(unsigned *words, uint64_t tile, unsigned sum, unsigned last) {
    const unsigned payload = last << 13 | sum;
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(words + tile * kStride), "r"(payload << 1 | 1u)
                 : "memory");
}
__device__ __forceinline__ unsigned rd_peek(const unsigned *w) {
    unsigned x;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(w) : "memory");
    return x;
}

// What a tile needs from the words before it, by the output half: `base` =
// the sum over the rounds before, `lower` = over the round's tiles before the
// CTA's; kLast: `last` = the latest position before the tile (row + 1).
template <bool kLast, unsigned kStride = kRdWordStride>
struct RdPrefix {
    const unsigned *words;
    uint64_t ntiles;
    uint64_t base = 0, last = 0;
    unsigned lower = 0;
    unsigned cur = 0, nxt = 0;
    unsigned total = 0;       // of the round
    uint64_t base_last = 0;   // latest position in the rounds before

    __device__ RdPrefix(const unsigned *w, uint64_t n) : words(w), ntiles(n) {}

    __device__ __forceinline__ unsigned in_round(unsigned r) const {
        return unsigned(minu(gridDim.x, ntiles - uint64_t(r) * gridDim.x));
    }
    __device__ __forceinline__ const unsigned *word(unsigned r, unsigned i) const {
        return words + (uint64_t(r) * gridDim.x + i) * kStride;
    }
    // requests round r's words; they are read by the next call of sums
    __device__ __forceinline__ void request(unsigned r, unsigned tid) {
        nxt = tid < in_round(r) ? rd_peek(word(r, tid)) : 1u;
    }
    __device__ __forceinline__ void sums(RdShared &sh, unsigned r, unsigned tid) {
        const unsigned n = in_round(r);
        unsigned lo = 0, to = 0, llo = 0, lto = 0;
        for (unsigned i = tid; i < n; i += kRdHalf) {
            unsigned x = i == tid ? cur : 0u;
            for (unsigned spins = 0; !(x & 1u) && !sh.fail; spins++) {
                if (spins >= kSpinLimit) sh.fail = 1;
                x = rd_peek(word(r, i));
            }
            const unsigned sum = (x >> 1) & 0x1FFFu, at = x >> 14 ? i << 13 | x >> 14 : 0u;
            to += sum;
            lo += i < blockIdx.x ? sum : 0u;
            lto = max(lto, at);
            llo = max(llo, i < blockIdx.x ? at : 0u);
        }
        lo = __reduce_add_sync(0xFFFFFFFFu, lo);
        to = __reduce_add_sync(0xFFFFFFFFu, to);
        if (kLast) {
            llo = __reduce_max_sync(0xFFFFFFFFu, llo);
            lto = __reduce_max_sync(0xFFFFFFFFu, lto);
        }
        if ((tid & 31u) == 0) {
            sh.lower[tid >> 5] = lo;
            sh.total[tid >> 5] = to;
            if (kLast) {
                sh.lower_last[tid >> 5] = llo;
                sh.total_last[tid >> 5] = lto;
            }
        }
        rd_bar(1);
        lower = total = 0;
        llo = lto = 0;
#pragma unroll
        for (unsigned i = 0; i < kRdWarps; i++) {
            lower += sh.lower[i];
            total += sh.total[i];
            if (kLast) {
                llo = max(llo, sh.lower_last[i]);
                lto = max(lto, sh.total_last[i]);
            }
        }
        if (kLast) {
            const auto row1 = [&](unsigned at) { return (uint64_t(r) * gridDim.x + (at >> 13)) * kRdRows + (at & 0x1FFFu); };
            last = llo ? row1(llo) : base_last;
            if (lto) base_last = row1(lto);
        }
    }
    __device__ __forceinline__ void next() { base += total; }
    // the requested words become the ones that sums reads
    __device__ __forceinline__ void turn() { cur = nxt; }
};

}  // namespace
}  // namespace ms
