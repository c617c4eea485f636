// positions.cuh -- operators that produce ascending row positions (select,
// semi_join, natural_join), in two launches without a scan between them.
//
// Pass 1 decides every row once and writes one bit per row (64 bytes per
// 512-row block, in row order) and the hit count of every unit of blocks.
// Pass 2 expands the bits: each CTA takes one unit, adds up the counts of the
// units before it (at most kMaxUnits) and writes its rows' positions.  The
// values are decoded once: the bits cost 1/8 byte per row written and read,
// decoding the column again its whole compressed size and the comparison.
//
// The bits live at the top of the arena for the time of the call (every call
// ends with the stream drained), so a call leaves only its positions behind.
//
// Measured against counting, scanning and deciding every row again in the
// second pass, both passes and the scan: select of 10% of 2^26 rows (for_f,
// 16 bits) 338 -> 105 us, semi_join of 2^26 rows (20-bit keys, bitmap of
// 2^20) 1006 -> 138 us, natural_join of 2^25 rows (half of them hit) 392 ->
// 244 us.  Pass 1 is bound by decoding and look-ups, pass 2 by its writes.
#pragma once

#include "fastpath.cuh"
#include "internal.h"
#include "readback.cuh"

namespace ms {
namespace {

constexpr unsigned kMaxUnits = 2048;     // counts that a pass-2 CTA may have to add up
constexpr unsigned kUnitWords = 256;     // bit words that a pass-2 CTA expands per step (16 blocks)
constexpr unsigned kCtaUnits = 32;       // units that one pass-1 CTA may touch
constexpr unsigned kBlockWords = kBlock / 32;

// The blocks of a pass: [b0, b0 + nblk) of the column, in units of `unit`
// blocks (a multiple of 16); bits and counts are indexed from b0.
struct MaskRun {
    uint64_t b0, nblk;
    unsigned unit, nunits;
    uint32_t *bits;
    unsigned *counts;  // hits per unit, zero before pass 1
};

inline unsigned mask_unit(uint64_t nblk) {
    const uint64_t per = uint64_t(16) * kMaxUnits;
    return unsigned(16 * maxu(1, (nblk + per - 1) / per));
}

// Row-order words of a block's hits (bit k of thread (l, q): row
// (16q + k) * 8 + l).  Word 4q + j holds the bits 4j .. 4j+3 of the eight
// threads of quarter q, byte by byte; the four words of a quarter are
// combined over its threads by a reduce-scatter (four shuffles), after which
// thread l < 4 holds word 4q + j(l).
__device__ __forceinline__ unsigned mask_word_of(unsigned l) { return ((l & 1u) << 1) | ((l >> 1) & 1u); }

__device__ __forceinline__ uint32_t mask_words(unsigned m, unsigned l) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = ((((m >> (4 * j)) & 15u) * 0x00204081u) & 0x01010101u) << l;
    const bool b0 = l & 1u, b1 = l & 2u;
    uint32_t x = b0 ? w[2] : w[0], y = b0 ? w[3] : w[1];
    x |= __shfl_xor_sync(0xFFFFFFFFu, b0 ? w[0] : w[2], 1);
    y |= __shfl_xor_sync(0xFFFFFFFFu, b0 ? w[1] : w[3], 1);
    uint32_t z = b1 ? y : x;
    z |= __shfl_xor_sync(0xFFFFFFFFu, b1 ? x : y, 2);
    return z | __shfl_xor_sync(0xFFFFFFFFu, z, 4);
}

// Pass 1 skeleton: the CTA's share of the blocks, one warp per block;
// hits(b, l, q) returns the thread's hit bits of block b of the column.
template <class Hits>
__device__ __forceinline__ void mask_pass(const MaskRun &r, Hits hits) {
    __shared__ unsigned s_cnt[kCtaUnits];
    if (threadIdx.x < kCtaUnits) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3, W = blockDim.x / 32u;
    const uint64_t lo = r.nblk * blockIdx.x / gridDim.x, hi = r.nblk * (blockIdx.x + 1) / gridDim.x;
    const unsigned u0 = unsigned(lo / r.unit);
    for (uint64_t i = lo + threadIdx.x / 32u; i < hi; i += W) {
        const unsigned m = hits(r.b0 + i, l, q);
        const uint32_t w = mask_words(m, l);
        if (l < 4) r.bits[i * kBlockWords + 4u * q + mask_word_of(l)] = w;
        const unsigned c = __reduce_add_sync(0xFFFFFFFFu, __popc(m));
        if (lane == 0 && c) atomicAdd(&s_cnt[unsigned(i / r.unit) - u0], c);
    }
    __syncthreads();
    if (threadIdx.x < kCtaUnits && s_cnt[threadIdx.x]) atomicAdd(r.counts + u0 + threadIdx.x, s_cnt[threadIdx.x]);
}

// Grid of pass 1: at least 2048 / 30 CTAs for a long column keeps a CTA's
// units within kCtaUnits; short columns have one block per warp.
inline unsigned mask_grid(uint64_t nblk, unsigned warps, unsigned ctas_per_sm) {
    return (unsigned)maxu(1, minu((nblk + warps - 1) / warps, maxu(persistent_grid(32 * warps, ctas_per_sm), 128)));
}

// What an operator gives per hit: the row's position, a value of its own
// (compact per block in `side`), or both.
enum : int { kRows = 1, kVals = 2 };

// Pass 2: positions and / or the compact per-block values of pass 1 (block
// i's j-th hit at side[i * 512 + j]) from *base_in on; the last unit
// stores the end in *base_out.  Words with many hits are written by a warp
// each (consecutive lanes, consecutive addresses), sparse ones by a lane
// each.  Nothing is written at or beyond index `cap`.  scalar: hits at rows
// >= sfrom.
template <int kOut, class V>
__global__ void __launch_bounds__(256) k_expand_rows(MaskRun r, uint64_t n, uint64_t sfrom,
                                                    const unsigned long long *__restrict__ base_in,
                                                    unsigned long long *__restrict__ base_out, uint64_t cap,
                                                    uint64_t *__restrict__ out, const V *__restrict__ side,
                                                    uint64_t *__restrict__ out_vals,
                                                    unsigned long long *__restrict__ scalar) {
    __shared__ unsigned long long s_sum[8];
    __shared__ unsigned s_w[8];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long before = 0;
    for (unsigned u = threadIdx.x; u < blockIdx.x; u += 256) before += r.counts[u];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, d);
    if (lane == 0) s_sum[warp] = before;
    __syncthreads();
    uint64_t base = *base_in;
#pragma unroll
    for (int w = 0; w < 8; w++) base += s_sum[w];
    if (base_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *base_out = base + r.counts[blockIdx.x];
    unsigned long long scal = 0;
    const uint64_t i0 = uint64_t(blockIdx.x) * r.unit, i1 = minu(r.nblk, i0 + r.unit);
    for (uint64_t w0 = i0 * kBlockWords; w0 < i1 * kBlockWords; w0 += kUnitWords) {
        const uint64_t wi = w0 + threadIdx.x;
        const uint32_t word = wi < i1 * kBlockWords ? __ldg(r.bits + wi) : 0u;
        const unsigned c = __popc(word);
        unsigned incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (int(lane) >= d) incl += o;
        }
        const unsigned wtot = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (lane == 0) s_w[warp] = wtot;
        __syncthreads();
        unsigned pre = 0, tot = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            pre += w < int(warp) ? s_w[w] : 0u;
            tot += s_w[w];
        }
        __syncthreads();
        const uint64_t wbase = base + pre;             // the warp's first output
        const uint64_t row = r.b0 * kBlock + wi * 32;  // the word's first row
        if (wtot && wbase + wtot <= cap) {
            if (!(kOut & kRows)) {
            } else if (wtot > 128) {
#pragma unroll 4
                for (int i = 0; i < 32; i++) {
                    const uint32_t x = __shfl_sync(0xFFFFFFFFu, word, i);
                    const unsigned o = __shfl_sync(0xFFFFFFFFu, incl - c, i);
                    if ((x >> lane) & 1u)
                        out[wbase + o + __popc(x & ((1u << lane) - 1u))] = row - 32ull * lane + 32ull * i + lane;
                }
            } else {
                uint64_t *o = out + wbase + (incl - c);
                for (uint32_t x = word; x; x &= x - 1) *o++ = row + unsigned(__ffs(x) - 1);
            }
            if (kOut & kVals) {
                // the warp's two blocks
                const unsigned c0 = __shfl_sync(0xFFFFFFFFu, incl, 15), c1 = wtot - c0;
                const V *s = side + (w0 + 32ull * warp) / kBlockWords * kBlock;
                for (unsigned j = lane; j < c0; j += 32) out_vals[wbase + j] = s[j];
                for (unsigned j = lane; j < c1; j += 32) out_vals[wbase + c0 + j] = s[kBlock + j];
            }
        }
        if (row + 32 > sfrom && word) {
            const uint32_t x = row >= sfrom ? word : word & (0xFFFFFFFFu << unsigned(sfrom - row));
            scal += __popc(x);
        }
        base += tot;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) scal += __shfl_xor_sync(0xFFFFFFFFu, scal, d);
    if (lane == 0 && scal) atomicAdd(scalar, scal);
}

// Scratch taken from the top of the arena for the time of a call.
struct TopScratch {
    ms_arena *a;
    uint64_t top;
    explicit TopScratch(ms_arena *arena) : a(arena), top(arena->cap / 256 * 256) {}
    uint64_t room() const {
        const uint64_t lo = align_up(a->used, 256);
        return top > lo ? top - lo : 0;
    }
    template <class T> T *take(uint64_t count) {
        const uint64_t bytes = align_up(maxu(count * sizeof(T), 1), 256);
        if (bytes > room()) return nullptr;
        top -= bytes;
        return reinterpret_cast<T *>(a->base + top);
    }
};

// The driver.  pass1(run, side): launches pass 1 over run's blocks.  The bits
// (and side values) of all blocks at once while they fit the free part of the
// arena, else the largest segments of blocks that do.  A single output is
// written into what is left and trimmed; two outputs, and a single one that
// does not fit beside the scratch or comes in segments, are counted first, so
// that they are exactly as long as they have to be and the scratch takes the
// rest: a call fails only when the results and the scratch of one block do
// not fit.  Segments cost a second pass 1 and two launches each: 2^21 rows with
// 100 hits take 0.05 ms (intersect_sorted) and 0.11 ms (natural_join) at once,
// 4.3 and 7.8 ms in 380 and 190 segments.
template <int kOut, class V, class Pass1>
int rows_by_mask(const ColView &x, Pass1 pass1, uint64_t **d_pos, uint64_t **d_vals, uint64_t *count,
                 uint64_t *n_scalar, ms_arena *a, cudaStream_t st) {
    const uint64_t nbt = x.nblocks_total(), n = x.n;
    constexpr bool kBoth = kOut == (kRows | kVals);
    constexpr uint64_t kSide = kOut & kVals ? kBlock * sizeof(V) : 0;  // bytes per block
    const uint64_t room = TopScratch(a).room();
    const auto units = [](uint64_t seg) { return (seg + mask_unit(seg) - 1) / mask_unit(seg) + 1; };
    // running base (two words), remainder hits; then the units' counts
    const auto head_words = [&](uint64_t seg) { return 4 + (units(seg) + 1) / 2; };
    const auto bytes = [&](uint64_t seg) {
        return align_up(8 * head_words(seg), 256) + align_up(maxu(4 * kBlockWords * seg, 1), 256) +
               (kSide ? align_up(maxu(kSide * seg, 1), 256) : 0);
    };
    const auto largest = [&](uint64_t avail) {
        uint64_t seg = minu(nbt, avail / (4 * kBlockWords + kSide));
        while (seg && bytes(seg) > avail) seg--;
        return seg;
    };
    uint64_t seg = 0;
    unsigned unit = 0;
    unsigned long long *words = nullptr;
    unsigned *counts = nullptr;
    uint32_t *bits = nullptr;
    V *side = nullptr;
    bool clean = false;  // the counts are zero
    // places the scratch for segments of up to `blocks` blocks
    const auto place = [&](uint64_t blocks) -> int {
        seg = blocks;
        if ((nbt && !seg) || bytes(seg) > room) return ms_fail(MS_ERR_NOMEM, "arena exhausted (positions)");
        unit = mask_unit(seg);
        TopScratch ts(a);
        words = ts.take<unsigned long long>(head_words(seg));
        counts = reinterpret_cast<unsigned *>(words + 4);
        bits = ts.take<uint32_t>(seg * kBlockWords);
        side = kSide ? ts.take<V>(seg * kBlock) : nullptr;
        MS_CUDA_TRY(cudaMemsetAsync(words, 0, 32 + 4 * units(seg), st));
        clean = true;
        return MS_OK;
    };
    const auto run_of = [&](uint64_t b0) {
        MaskRun r{b0, minu(seg, nbt - b0), unit, 0, bits, counts};
        r.nunits = unsigned((r.nblk + unit - 1) / unit);
        return r;
    };
    const auto first = [&](const MaskRun &r) -> int {
        if (!clean) MS_CUDA_TRY(cudaMemsetAsync(counts, 0, 4 * r.nunits, st));
        clean = false;
        pass1(r, side);
        MS_CUDA_TRY(cudaGetLastError());
        return MS_OK;
    };
    uint64_t *pos = nullptr, *vals = nullptr;
    // pass 2 (and, unless the bits are there already, pass 1) of every segment;
    // hw: the end of the results in hw[0] or hw[1], remainder hits in hw[2]
    const auto expand = [&](uint64_t cap, bool have_bits, const unsigned long long **hw, uint64_t *end) -> int {
        unsigned ping = 0;
        for (uint64_t b0 = 0; b0 < nbt; b0 += seg, ping ^= 1u) {
            const MaskRun r = run_of(b0);
            if (!have_bits) {
                int rc = first(r);
                if (rc) return rc;
            }
            k_expand_rows<kOut, V><<<r.nunits, 256, 0, st>>>(r, n, x.sfrom, words + ping, words + (ping ^ 1u), cap, pos,
                                                              side, vals, words + 2);
            MS_CUDA_TRY(cudaGetLastError());
        }
        ReadBack back(a, st);
        *hw = back.add(words, 3);
        int rc = back.wait();
        if (!rc) *end = (*hw)[ping];
        return rc;
    };
    int rc = place(bytes(nbt) <= room ? nbt : largest(room));
    if (rc) return rc;
    uint64_t total = 0;
    const unsigned long long *hw = nullptr;
    bool done = false, have_bits = false;
    if (!kBoth && seg == nbt) {
        pos = vals = reinterpret_cast<uint64_t *>(a->base + align_up(a->used, 256));
        const uint64_t cap = minu(n, (room - bytes(seg)) / 8);
        rc = expand(cap, false, &hw, &total);
        if (rc) return rc;
        done = total <= cap;
    } else {
        for (uint64_t b0 = 0; b0 < nbt; b0 += seg) {
            const MaskRun r = run_of(b0);
            rc = first(r);
            if (rc) return rc;
            ReadBack back(a, st);
            const unsigned *h = back.add(counts, r.nunits);
            rc = back.wait_results();
            if (rc) return rc;
            for (unsigned u = 0; u < r.nunits; u++) total += h[u];
        }
        have_bits = seg == nbt;
    }
    if (!done) {
        const uint64_t one = 8 * (total + 1), results = kBoth ? align_up(one, 256) + one : one;
        if (results > room) return ms_fail(MS_ERR_NOMEM, "arena exhausted (positions output)");
        if (!have_bits || bytes(seg) + results > room) {
            have_bits = false;
            rc = place(largest(room - results));
            if (rc) return rc;
        }
    }
    const uint64_t mark = a->used;
    uint64_t *const out0 = arena_take_t<uint64_t>(a, total + 1), *const out1 = kBoth ? arena_take_t<uint64_t>(a, total + 1) : out0;
    if (!out0 || !out1) {
        a->used = mark;
        return ms_fail(MS_ERR_NOMEM, "arena exhausted (positions output)");
    }
    pos = out0;
    vals = out1;
    if (!done) {
        uint64_t end = 0;
        rc = expand(total, have_bits, &hw, &end);
        if (rc) return rc;
    }
    if (kOut & kRows) *d_pos = pos;
    if (kOut & kVals) *d_vals = vals;
    *count = total;
    *n_scalar = hw[2];
    return MS_OK;
}

// Smallest and largest value of a column: mn starts at ~0, nmx (the minimum of
// the complements) too.
__global__ void __launch_bounds__(256) k_key_range(ColView c, unsigned long long *mn, unsigned long long *nmx,
                                                  unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    uint64_t lo = ~uint64_t(0), hi = 0;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < c.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16];
        unsigned valid;
        ok &= decode_block(c, b, l, q, v, valid);
#pragma unroll
        for (int k = 0; k < 16; k++)
            if ((valid >> k) & 1u) {
                lo = minu(lo, v[k]);
                hi = maxu(hi, v[k]);
            }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
    // one atomic pair per CTA (one per thread queued up on the two words)
    __shared__ unsigned long long s_lo[8], s_hi[8];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        lo = minu(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, d));
        hi = maxu(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, d));
    }
    if (lane == 0) {
        s_lo[threadIdx.x >> 5] = lo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < blockDim.x / 32; w++) {
            lo = minu(lo, s_lo[w]);
            hi = maxu(hi, s_hi[w]);
        }
        atomicMin(mn, (unsigned long long)lo);
        atomicMin(nmx, ~(unsigned long long)hi);
    }
}

// [*lo, *hi] of a non-empty column's values (synchronises the stream); two
// device words as scratch.
inline int key_range(const ColView &c, unsigned long long *words, uint64_t *lo, uint64_t *hi, ms_arena *a,
                     cudaStream_t st) {
    MS_CUDA_TRY(cudaMemsetAsync(words, 0xFF, 16, st));
    const uint64_t nb = c.nblocks_total();
    k_key_range<<<unsigned(maxu(1, minu((nb + 7) / 8, persistent_grid(256, 8)))), 256, 0, st>>>(c, words, words + 1,
                                                                                                a->d_err);
    MS_CUDA_TRY(cudaGetLastError());
    ReadBack back(a, st);
    const unsigned long long *h = back.add(words, 2);
    int rc = back.wait_results();
    if (rc) return rc;
    *lo = h[0];
    *hi = ~h[1];
    return MS_OK;
}

}  // namespace
}  // namespace ms
