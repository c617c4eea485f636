// codecs.cu -- compression and decompression kernels for every format and
// the column-level morph (morph.h:81-241).
//
// Encoding a dynamic_vbp-family column is one pass in rounds (rounds.cuh):
// a tile of 12 blocks is staged in shared memory, its block widths found
// (OR-reduce, dynamic_vbp.h:124-158) after the cascade transform (delta:
// x[i]-x[i-8], delta.h:107-156; for: minus the block minimum,
// for.h:121-161), and once the widths before it are known the blocks are
// packed in place and copied to their offsets -- 64 * (headers before the
// block) + 64 * (sum of earlier widths) -- with page headers (bit-width bytes /
// 0xFF, FOR reference words) and block index entries.
// The same encoder writes operator outputs with the write iterator's
// 2048-value chunking (write_iterator.h:67-306): only the number of blocks
// per page changes (64 -> 4 for dynamic_vbp, 8 -> 2 for for_f).
#include <cuda.h>
#include <string.h>

#include "delta.cuh"
#include "fastpath.cuh"
#include "internal.h"
#include "readback.cuh"
#include "rounds.cuh"
#include "scan.cuh"
#include "tma.cuh"

namespace ms {
namespace {

struct Layout {
    int fmt;
    unsigned bw;          // static_vbp
    unsigned dvbp_shift;  // log2 of blocks per dynamic_vbp page (6 morph, 2 write iterator)
    unsigned for_shift;   // log2 of cascade blocks per for_f page (3 morph, 1 write iterator)
};

// 64-B headers preceding block b's packed data.
template <int FMT>
__device__ __forceinline__ uint64_t headers_before(const Layout &L, uint64_t b) {
    switch (FMT) {
    case MS_FMT_DYNAMIC_VBP: return (b >> L.dvbp_shift) + 1;
    case MS_FMT_DELTA_DVBP: return b / 2 + 1;
    default: return (b >> (1 + L.for_shift)) + 1 + b / 2 + 1;
    }
}

// --- packing: static_vbp ------------------------------------------------------
// Eight threads per block, one per lane stream; a warp packs four blocks.
__global__ void __launch_bounds__(256) k_pack_static(const uint64_t *__restrict__ in, uint64_t nb, unsigned bw,
                                                    uint8_t *__restrict__ out, unsigned *err) {
    const unsigned l = threadIdx.x & 7u;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 8; b < nb;
         b += uint64_t(gridDim.x) * blockDim.x / 8) {
        const uint64_t *blk = in + b * kBlock;
        auto get = [&](unsigned v) -> uint64_t { return __ldg(blk + v * 8 + l); };
        if (!vbp_pack_lane_rt(bw, get, reinterpret_cast<uint64_t *>(out + b * 64ull * bw), l)) atomicOr(err, kErrCorrupt);
    }
}

// --- dynamic_vbp family: one pass in rounds -----------------------------------
// Packing: thread (l, h) of a half-warp holds values 32h .. 32h+31 of lane l's
// stream of a block; they are exactly BW 32-bit words of the packed stream.
// dst: the block's first byte in shared memory.
template <unsigned BW>
__device__ __forceinline__ void pack_half(const uint64_t (&x)[32], uint8_t *dst, unsigned l, unsigned h) {
    uint32_t w[BW];
#pragma unroll
    for (unsigned j = 0; j < BW; j++) w[j] = 0;
#pragma unroll
    for (unsigned v = 0; v < 32; v++) {
        const uint32_t lo = uint32_t(x[v]), hi = uint32_t(x[v] >> 32);
        const unsigned bit = v * BW, wi = bit >> 5, sh = bit & 31u;
        w[wi] |= lo << sh;
        if (BW <= 32) {
            if (sh + BW > 32) w[wi + 1] |= lo >> (32 - sh);
        } else {
            w[wi + 1] |= __funnelshift_l(lo, hi, sh);
            if (sh + BW > 64) w[wi + 2] |= hi >> (32 - sh);
        }
    }
    uint8_t *o = dst + 8u * l + h * (BW / 2) * 64u;
    if (BW % 2 == 0) {
#pragma unroll
        for (unsigned j = 0; j < BW; j += 2)
            *reinterpret_cast<uint64_t *>(o + 32u * j) = uint64_t(w[j + (j + 1 < BW ? 1 : 0)]) << 32 | w[j];
    } else {
        // the second half starts in the middle of a 64-bit word
#pragma unroll
        for (unsigned j = 0; j < BW; j++)
            *reinterpret_cast<uint32_t *>(o + (h ? ((j + 1) >> 1) * 64u + ((j + 1) & 1u) * 4u
                                                 : (j >> 1) * 64u + (j & 1u) * 4u)) = w[j];
    }
}

__device__ __forceinline__ void pack_half_rt(unsigned bw, const uint64_t (&x)[32], uint8_t *dst, unsigned l, unsigned h) {
    switch (bw) {
#define MS_X(B) \
    case B: pack_half<B>(x, dst, l, h); break;
        MS_BW_CASES(MS_X)
#undef MS_X
    default: break;  // widths come from effective_bitwidth
    }
}

constexpr unsigned kEncBlocks = kRdRows / kBlock;  // 12 blocks per tile, two per warp
// rest rows that the last tile's warps copy themselves
constexpr uint64_t kEncRest = 4096;

template <int FMT>
__global__ void __launch_bounds__(kRdThreads, 1)
    k_encode(const uint64_t *__restrict__ in, uint64_t nb, Layout L, unsigned *words, uint8_t *__restrict__ out,
             uint64_t *__restrict__ index, uint64_t *__restrict__ refs, uint64_t nrest, uint64_t *__restrict__ d_compr,
             unsigned *err) {
    extern __shared__ __align__(128) uint8_t rd_smem[];
    __shared__ RdShared sh;
    __shared__ unsigned s_bw[kRdBufs][kEncBlocks];  // by buffer
    __shared__ uint64_t s_ref[kRdBufs][kEncBlocks / 2];
    const unsigned tid = threadIdx.x % kRdHalf, w = tid >> 5, lane = tid & 31u;
    const unsigned l = lane & 7u, h = (lane >> 3) & 1u, half = lane >> 4, j = 2 * w + half;
    const bool first_half = threadIdx.x < kRdHalf;
    const uint64_t ntiles = (nb + kEncBlocks - 1) / kEncBlocks;
    const unsigned rounds = unsigned((ntiles + gridDim.x - 1) / gridDim.x);
    auto tile_of = [&](unsigned r) { return uint64_t(r) * gridDim.x + blockIdx.x; };
    auto blocks_of = [&](uint64_t t) { return unsigned(minu(kEncBlocks, nb - t * kEncBlocks)); };
    auto load = [&](unsigned r) {
        const uint64_t t = tile_of(r);
        if (t < ntiles)
            rd_load(rd_buf(rd_smem, r), sh.full + r % kRdBufs, in, t * kRdRows, blocks_of(t) * kBlock,
                    FMT == MS_FMT_DELTA_DVBP && t ? 8u : 0u);
    };
    rd_init(sh);
    if (threadIdx.x == 0) {
        for (unsigned r = 0; r < kRdBufs; r++) load(r);
    }
    RdPrefix<false> pre(words, ntiles);
    for (unsigned r = 0; r <= rounds + 1; r++) {
        const uint64_t t = tile_of(r);
        if (first_half && t < ntiles) {
            const unsigned nblk = blocks_of(t), par = r % kRdBufs;
            const bool mine = j < nblk;
            uint8_t *const blk = rd_buf(rd_smem, r) + rd_row(kBlock * j);
            rd_full(sh, r);
            // The thread's 32 values.  The two halves read the values of a
            // pair in opposite order: halves and blocks lie a multiple of 128
            // bytes apart, so that in the same order all four groups of eight
            // threads would meet in the same banks.
            uint64_t x[32], acc = 1;
            {
                const uint8_t *const v0 = blk + 8u * (256u * h + l);
                const uint8_t *const p0 = v0 + 64u * h, *const p1 = v0 + 64u - 64u * h;
#pragma unroll
                for (unsigned v = 0; v < 32; v += 2) {
                    const uint64_t a = mine ? *reinterpret_cast<const uint64_t *>(p0 + 64u * v) : 0;
                    const uint64_t b = mine ? *reinterpret_cast<const uint64_t *>(p1 + 64u * v) : 0;
                    x[v] = h ? b : a;
                    x[v + 1] = h ? a : b;
                }
                if (FMT == MS_FMT_DELTA_DVBP) {
                    const bool none = !mine || (t == 0 && j == 0 && h == 0);  // the column's first rows
                    const uint64_t prev = none ? 0 : *reinterpret_cast<const uint64_t *>(v0 - 64);
#pragma unroll
                    for (int v = 31; v > 0; v--) x[v] -= x[v - 1];
                    x[0] -= prev;
                }
            }
            if (FMT == MS_FMT_FOR_DVBP) {
                // the warp's pair is one 1024-block; its reference is the
                // AVX-512 TVL minimum (signed per lane, _mm512_min_epi64, then
                // unsigned across lanes; for.h:121-161); l is the TVL lane
                int64_t mn = INT64_MAX;
#pragma unroll
                for (unsigned v = 0; v < 32; v++) mn = min(mn, (int64_t)x[v]);
                mn = min(mn, (int64_t)__shfl_xor_sync(0xFFFFFFFFu, (uint64_t)mn, 8));
                mn = min(mn, (int64_t)__shfl_xor_sync(0xFFFFFFFFu, (uint64_t)mn, 16));
                uint64_t um = (uint64_t)mn;
                um = minu(um, __shfl_xor_sync(0xFFFFFFFFu, um, 1));
                um = minu(um, __shfl_xor_sync(0xFFFFFFFFu, um, 2));
                um = minu(um, __shfl_xor_sync(0xFFFFFFFFu, um, 4));
                if (um == ~uint64_t(0)) um--;
#pragma unroll
                for (unsigned v = 0; v < 32; v++) x[v] -= um;
                if (lane == 0 && mine) {
                    s_ref[par][w] = um;
                    refs[t * (kEncBlocks / 2) + w] = um;
                }
            }
#pragma unroll
            for (unsigned v = 0; v < 32; v++) acc |= x[v];
            // widths of the warp's two blocks
            const unsigned h0 = __reduce_or_sync(0xFFFFFFFFu, half ? 0u : unsigned(acc >> 32));
            const unsigned h1 = __reduce_or_sync(0xFFFFFFFFu, half ? unsigned(acc >> 32) : 0u);
            const unsigned l0 = __reduce_or_sync(0xFFFFFFFFu, half ? 0u : unsigned(acc));
            const unsigned l1 = __reduce_or_sync(0xFFFFFFFFu, half ? unsigned(acc) : 0u);
            const unsigned bw = effective_bitwidth(half ? uint64_t(h1) << 32 | l1 : uint64_t(h0) << 32 | l0);
            if ((lane & 15u) == 0 && mine) s_bw[par][j] = bw;
            rd_bar(0);  // every value of the tile is in registers
            if (w == kRdWarps - 1) {
                const unsigned sum = __reduce_add_sync(0xFFFFFFFFu, lane < nblk ? s_bw[par][lane] : 0u);
                if (lane == 0) rd_publish(words, t, sum, 0);
            }
            if (mine) pack_half_rt(bw, x, blk, l, h);
        }
        if (!first_half && r && r <= rounds) pre.request(r - 1, tid);  // read in the next round
        if (!first_half && r > 1) {
            // tile r - 2, packed in place, goes to its place, and its buffer
            // takes tile r + 2
            const uint64_t tp = tile_of(r - 2);
            pre.sums(sh, r - 2, tid);
            if (tp < ntiles) {
                const unsigned nblk = blocks_of(tp), par = (r - 2) % kRdBufs;
                const uint8_t *const stage = rd_buf(rd_smem, r - 2) + rd_row(kBlock * j);  // the half-warp's packed block
                const unsigned bl = lane < nblk ? s_bw[par][lane] : 0u;
                unsigned ex = bl;  // widths of the tile's blocks before each
    #pragma unroll
                for (int d = 1; d < 16; d <<= 1) {
                    const unsigned o = __shfl_up_sync(0xFFFFFFFFu, ex, d);
                    if (int(lane) >= d) ex += o;
                }
                const unsigned before = __shfl_sync(0xFFFFFFFFu, ex - bl, j), bwp = __shfl_sync(0xFFFFFFFFu, bl, j);
                const unsigned bw1 = __shfl_sync(0xFFFFFFFFu, bl, 2 * w + 1);  // 0 when the pair has one block
                const bool mine = j < nblk;
                const uint64_t b = tp * kEncBlocks + j;
                const uint64_t off = 64ull * headers_before<FMT>(L, b) + 64ull * (pre.base + pre.lower + before);
                if (mine) {
                    // 16 bytes per thread and step, four steps in flight
                    const uint4 *from = reinterpret_cast<const uint4 *>(stage);
                    uint4 *to = reinterpret_cast<uint4 *>(out + off);
                    for (unsigned i0 = lane & 15u; i0 < 4u * bwp; i0 += 64) {
                        uint4 q[4];
    #pragma unroll
                        for (unsigned i = 0; i < 4; i++)
                            if (i0 + 16u * i < 4u * bwp) q[i] = from[i0 + 16u * i];
    #pragma unroll
                        for (unsigned i = 0; i < 4; i++)
                            if (i0 + 16u * i < 4u * bwp) to[i0 + 16u * i] = q[i];
                    }
                    if ((lane & 15u) == 0) index[b] = idx_pack(off, bwp);
                }
                if (FMT == MS_FMT_DYNAMIC_VBP) {
                    // pages of at most four blocks: the header is written with
                    // the page's first block (larger pages: k_headers_dvbp)
                    const unsigned page = 1u << L.dvbp_shift;
                    if (page <= 4 && mine && (j & (page - 1)) == 0 && (lane & 15u) < 8) {
                        uint64_t word = ~uint64_t(0);
                        if ((lane & 7u) == 0)
                            for (unsigned i = 0; i < page && j + i < nblk; i++)
                                word = (word & ~(0xFFull << (8 * i))) | uint64_t(s_bw[par][j + i]) << (8 * i);
                        reinterpret_cast<uint64_t *>(out + off - 64)[lane & 7u] = word;
                    }
                } else if (mine && lane < 8) {
                    // inner dynamic_vbp header of the 1024-block: two widths,
                    // 62 x 0xFF
                    uint64_t word = ~uint64_t(0);
                    if (lane == 0) word = (~uint64_t(0) << 16) | uint64_t(bwp) | uint64_t(bw1) << 8;
                    reinterpret_cast<uint64_t *>(out + off - 64)[lane] = word;
                    const unsigned page = 1u << L.for_shift;
                    if (FMT == MS_FMT_FOR_DVBP && page <= 2 && (w & (page - 1)) == 0) {
                        // page header: references, end marker, zeros (larger
                        // pages: k_headers_for)
                        const unsigned nbp = min(page, nblk / 2 - w);
                        reinterpret_cast<uint64_t *>(out + off - 128)[lane] =
                            lane < nbp ? s_ref[par][w + lane] : lane == nbp ? ~uint64_t(0) : 0;
                    }
                }
                if (tp == ntiles - 1) {
                    // the column's end: the compressed size, a short rest behind it
                    const unsigned in_tile = __reduce_add_sync(0xFFFFFFFFu, bl);
                    const uint64_t compr = 64ull * headers_before<FMT>(L, nb - 1) + 64ull * (pre.base + pre.lower + in_tile);
                    if (tid == 0) *d_compr = compr;
                    if (nrest <= kEncRest) {
                        uint64_t *dst = reinterpret_cast<uint64_t *>(out + rest_offset(FMT, 0, compr));
                        for (unsigned i = tid; i < nrest; i += kRdHalf) dst[i] = __ldg(in + nb * kBlock + i);
                    }
                }
            }
            pre.next();
            fence_async_smem();  // the buffer's last accesses, before a bulk copy overwrites it
            rd_bar(1);
            if (tid == 0) load(r + 2);
        }
        if (first_half) fence_async_smem();
        else pre.turn();
        __syncthreads();
    }
    if (sh.fail && threadIdx.x == 0) atomicOr(err, kErrTimeout);
}

// Headers of dynamic_vbp pages longer than a tile: one thread per header byte.
__global__ void k_headers_dvbp(uint64_t nb, unsigned page, const uint64_t *__restrict__ index,
                               uint8_t *__restrict__ out) {
    const uint64_t pages = (nb + page - 1) / page;
    for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < pages * kPageBlocks;
         t += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t p = t / kPageBlocks, j = t % kPageBlocks, b = p * page + j;
        out[idx_off(index[p * page]) - 64 + j] = (j < page && b < nb) ? uint8_t(idx_bw(index[b])) : uint8_t(kNoBlock);
    }
}

// Headers of for_f pages longer than a tile: references, end marker, zeros.
__global__ void k_headers_for(uint64_t ncb, unsigned page, const uint64_t *__restrict__ index,
                              const uint64_t *__restrict__ refs, uint8_t *__restrict__ out) {
    const uint64_t pages = (ncb + page - 1) / page;
    for (uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; t < pages * 8; t += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t c = t / 8 * page, w = t % 8, nbp = minu(page, ncb - c);
        reinterpret_cast<uint64_t *>(out + idx_off(index[2 * c]) - 128)[w] =
            w < nbp ? refs[c + w] : w == nbp ? ~uint64_t(0) : 0;
    }
}

// Uncompressed rest: copied behind the gap (morph.h:186-189,
// write_iterator.h:157-170).  A compressed size known on the device only is
// read there.
__global__ void k_copy_rest(const uint64_t *__restrict__ in, uint64_t nrest, int fmt, unsigned bw,
                            const uint64_t *__restrict__ d_compr, uint64_t compr, uint8_t *__restrict__ out) {
    const uint64_t ro = rest_offset(fmt, bw, d_compr ? *d_compr : compr);
    uint64_t *dst = reinterpret_cast<uint64_t *>(out + ro);
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nrest; i += uint64_t(gridDim.x) * blockDim.x)
        dst[i] = in[i];
}

// --- decompression ------------------------------------------------------------
__global__ void __launch_bounds__(256, 3) k_decode_all(ColView c, uint64_t *__restrict__ out, unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    const uint64_t nbt = c.nblocks_total();
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < nbt;
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16];
        unsigned valid;
        if (!decode_block(c, b, l, q, v, valid) && lane == 0) atomicOr(err, kErrCorrupt);
        const uint64_t row0 = b * kBlock;
#pragma unroll
        for (int k = 0; k < 16; k++)
            if ((valid >> k) & 1u) out[row0 + (16u * q + k) * 8u + l] = v[k];
    }
}

// delta_f: one warp per segment of blocks, the lanes' carry in registers from
// block to block; running sums of up to 27-bit deltas in 32 bits.  The blocks
// behind the compressed part (uncompressed rows) follow the segments.  2^27
// rows of 9-bit deltas: 234 us, 188 at the copy rate; with the scan of every
// block's sums and the carries stored and read back the call took 367 us in
// kernels, now 311.
__global__ void __launch_bounds__(256, 3) k_decode_delta(ColView c, DeltaSegs g, uint64_t *__restrict__ out,
                                                        unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    const uint64_t nb = c.nb(), rest_blocks = c.nblocks_total() - nb;
    bool ok = true;
    for (uint64_t s = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; s < g.nseg + rest_blocks;
         s += uint64_t(gridDim.x) * blockDim.x / 32) {
        if (s >= g.nseg) {
            const uint64_t r0 = (nb + s - g.nseg) * kBlock;
            for (uint64_t r = r0 + lane; r < minu(c.n, r0 + kBlock); r += 32) out[r] = __ldg(c.rest + (r - c.n_compr));
            continue;
        }
        const uint64_t b0 = s * g.blocks, b1 = minu(nb, b0 + g.blocks);
        uint64_t carry = __ldg(g.prefix + s * 8 + l), e = __ldg(c.index + b0);
        for (uint64_t b = b0; b < b1; b++) {
            const uint64_t next = b + 1 < b1 ? __ldg(c.index + b + 1) : 0;
            const uint64_t *blk = reinterpret_cast<const uint64_t *>(c.data + idx_off(e));
            const unsigned bw = idx_bw(e);
            uint64_t *const o = out + b * kBlock + 128u * q + l;
            uint32_t p[16];
            uint64_t last;
            if (bw <= 27 && vbp_decode16_u32_rt(bw, blk, l, q, p)) {
#pragma unroll
                for (int k = 1; k < 16; k++) p[k] += p[k - 1];
                const uint64_t tot = p[15], up = __shfl_up_sync(0xFFFFFFFFu, tot, 8);
                uint64_t pre = q >= 1 ? up : 0;
                const uint64_t up2 = __shfl_up_sync(0xFFFFFFFFu, tot + pre, 16);
                pre += (q >= 2 ? up2 : 0) + carry;
#pragma unroll
                for (int k = 0; k < 16; k++) o[8 * k] = pre + p[k];
                last = pre + p[15];
            } else {
                uint64_t v[16];
                ok &= vbp_decode16_rt(bw, blk, l, q, v);
                apply_cascade(c, b, l, q, v, carry);
#pragma unroll
                for (int k = 0; k < 16; k++) o[8 * k] = v[k];
                last = v[15];
            }
            carry = __shfl_sync(0xFFFFFFFFu, last, int(24 + l));
            e = next;
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
}

// --- rle ----------------------------------------------------------------------
// Encoder: one pass in rounds (rounds.cuh).  A row starts a run (a "head") when
// it differs from the row before (rle.h:63-150: maximal runs).  The analysing
// warps find a tile's heads (one ballot per 32 rows) and publish their number
// and the last one; the writing warps get from the words before the tile the
// number of runs before it and the row where the run that its first head ends
// began.  Every head writes the pair of the run it ends (the value of the row
// before it, its length), the column's last tile also the final run.  So the
// input is read once and each pair written once (8 B/row + 16 B/run).  2^26
// rows, mean run 32: 149 us (208 with a look-back by CTAs that load, search,
// look back and write one after another; 87 at the copy rate); runs of one
// row 350 us a call (373), of 1000 rows 188 us (226).
template <unsigned kStride>
__global__ void __launch_bounds__(kRdThreads, 1)
    k_rle_encode(const uint64_t *__restrict__ in, uint64_t n, unsigned *words, ulonglong2 *__restrict__ out,
                 uint64_t *__restrict__ d_runs, unsigned *err) {
    extern __shared__ __align__(128) uint8_t rd_smem[];
    __shared__ RdShared sh;
    __shared__ unsigned s_heads[kRdBufs][kRdRows / 32];  // by buffer: heads of 32 rows
    __shared__ unsigned s_cnt[kRdWarps], s_last[kRdWarps];
    const unsigned tid = threadIdx.x % kRdHalf, w = tid >> 5, lane = tid & 31u;
    const bool first_half = threadIdx.x < kRdHalf;
    const uint64_t ntiles = (n + kRdRows - 1) / kRdRows;
    const unsigned rounds = unsigned((ntiles + gridDim.x - 1) / gridDim.x);
    auto tile_of = [&](unsigned r) { return uint64_t(r) * gridDim.x + blockIdx.x; };
    auto rows_of = [&](uint64_t t) { return unsigned(minu(kRdRows, n - t * kRdRows)); };
    auto load = [&](unsigned r) {
        const uint64_t t = tile_of(r);
        if (t < ntiles)
            rd_load(rd_buf(rd_smem, r), sh.full + r % kRdBufs, in, t * kRdRows, rows_of(t), t ? 2u : 0u);
    };
    rd_init(sh);
    if (threadIdx.x == 0) {
        for (unsigned r = 0; r < kRdBufs; r++) load(r);
    }
    RdPrefix<true, kStride> pre(words, ntiles);
    for (unsigned r = 0; r <= rounds + 1; r++) {
        const uint64_t t = tile_of(r);
        if (first_half && t < ntiles) {
            const unsigned rows = rows_of(t);
            uint64_t *const v = reinterpret_cast<uint64_t *>(rd_buf(rd_smem, r) + kRdHead);
            rd_full(sh, r);
            if (rows & 1u) {  // the column's odd last row
                if (tid == 0) v[rows - 1] = __ldg(in + n - 1);
                rd_bar(0);
            }
            // warp w: rows [1024 w, 1024 (w + 1)); lane k keeps word k
            unsigned mine = 0;
#pragma unroll 8
            for (unsigned k = 0; k < 32; k++) {
                const unsigned i = 1024u * w + 32u * k + lane;
                const bool head = i < rows && (t + i == 0 || v[i] != v[int(i) - 1]);
                const unsigned b = __ballot_sync(0xFFFFFFFFu, head);
                if (k == lane) mine = b;
            }
            s_heads[r % kRdBufs][32 * w + lane] = mine;
            const unsigned cnt = __reduce_add_sync(0xFFFFFFFFu, __popc(mine));
            const unsigned last = __reduce_max_sync(0xFFFFFFFFu, mine ? 1024u * w + 32u * lane + 32u - __clz(mine) : 0u);
            if (lane == 0) {
                s_cnt[w] = cnt;
                s_last[w] = last;
            }
            rd_bar(0);
            if (tid == 0) {
                unsigned c = 0, z = 0;
                for (unsigned i = 0; i < kRdWarps; i++) {
                    c += s_cnt[i];
                    z = max(z, s_last[i]);
                }
                rd_publish<kStride>(words, t, c, z);
            }
        }
        if (!first_half && r && r <= rounds) pre.request(r - 1, tid);  // read in the next round
        if (!first_half && r > 1) {
            const uint64_t tp = tile_of(r - 2);
            pre.sums(sh, r - 2, tid);
            if (tp < ntiles) {
                const uint64_t *const v = reinterpret_cast<const uint64_t *>(rd_buf(rd_smem, r - 2) + kRdHead);
                const unsigned *const heads = s_heads[(r - 2) % kRdBufs];
                // runs before the warp's first word, the head before it
                unsigned before = 0, prev = 0;  // prev: row of the tile + 1, 0 for none in the tile
                for (unsigned i = lane; i < 32 * w; i += 32) {
                    const unsigned x = heads[i];
                    before += __popc(x);
                    if (x) prev = 32u * i + 32u - __clz(x);
                }
                before = __reduce_add_sync(0xFFFFFFFFu, before);
                prev = __reduce_max_sync(0xFFFFFFFFu, prev);
                const unsigned word = heads[32 * w + lane], c = __popc(word);
                unsigned incl = c, lastw = word ? 1024u * w + 32u * lane + 32u - __clz(word) : 0u;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const unsigned o = __shfl_up_sync(0xFFFFFFFFu, incl, d), z = __shfl_up_sync(0xFFFFFFFFu, lastw, d);
                    if (int(lane) >= d) {
                        incl += o;
                        lastw = max(lastw, z);
                    }
                }
                const unsigned tot = __shfl_sync(0xFFFFFFFFu, incl, 31), tail = max(prev, __shfl_sync(0xFFFFFFFFu, lastw, 31));
                unsigned ph = __shfl_up_sync(0xFFFFFFFFu, lastw, 1);  // the head before the lane's word
                ph = max(prev, lane ? ph : 0u);
                const uint64_t row0 = tp * kRdRows, run0 = pre.base + pre.lower + before;
                // the pair that the head at tile row i ends: run `run` of the
                // column, which began at the head before, p (+ 1, 0: before the tile)
                auto put = [&](uint64_t run, unsigned i, unsigned p) {
                    if (run) out[run - 1] = make_ulonglong2(v[int(i) - 1], row0 + i + 1 - (p ? row0 + p : pre.last));
                };
                if (__reduce_max_sync(0xFFFFFFFFu, c) > 20) {
                    // nearly all rows are heads: a warp per word, consecutive
                    // lanes write consecutive pairs; else a lane per word,
                    // which takes as many steps as its word has heads
                    for (unsigned k = 0; k < 32; k++) {
                        const unsigned x = __shfl_sync(0xFFFFFFFFu, word, k), o = __shfl_sync(0xFFFFFFFFu, incl - c, k);
                        const unsigned p = __shfl_sync(0xFFFFFFFFu, ph, k), below = x & ((1u << lane) - 1u);
                        const unsigned i = 1024u * w + 32u * k;
                        if ((x >> lane) & 1u) put(run0 + o + __popc(below), i + lane, below ? i + 32u - __clz(below) : p);
                    }
                } else {
                    uint64_t run = run0 + (incl - c);
                    unsigned p = ph;
                    for (unsigned x = word; x; x &= x - 1) {
                        const unsigned i = 1024u * w + 32u * lane + unsigned(__ffs(x) - 1);
                        put(run++, i, p);
                        p = i + 1;
                    }
                }
                if (tp == ntiles - 1 && w == kRdWarps - 1 && lane == 0) {
                    // the final run ends at row n
                    const uint64_t total = run0 + tot;
                    uint64_t slot;
                    *d_runs = total;
                    if (rle_last_slot(total, n, slot))
                        out[slot] = make_ulonglong2(v[n - row0 - 1], n + 1 - (tail ? row0 + tail : pre.last));
                }
            }
            pre.next();
            fence_async_smem();  // the buffer's last accesses, before a bulk copy overwrites it
            rd_bar(1);
            if (tid == 0) load(r + 2);
        }
        if (first_half) fence_async_smem();
        else pre.turn();
        __syncthreads();
    }
    if (sh.fail && threadIdx.x == 0) atomicOr(err, kErrTimeout);
}

// The short-run decoder's tiles find the rows before them by a decoupled
// look-back over the tiles before (every tile publishes its own row count,
// then -- once known -- the inclusive one).
// A tile's published count carries the flag in its low two bits (0: nothing
// yet, kRleFlagAgg: the tile's own rows, kRleFlagInc: the rows of tiles [0,
// this tile]): written and read whole, so no fence is needed.  It has a cache
// line of its own (rounds.cuh) unless the arena is short: `stride` words from
// one tile's to the next.
enum : unsigned { kRleFlagAgg = 1, kRleFlagInc = 2 };
constexpr unsigned kRleStateStride = 16;

__device__ __forceinline__ void rle_publish(unsigned long long *s, unsigned flag, uint64_t rows) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(s), "l"((rows << 2) | flag) : "memory");
}

// Warp-wide look-back (warp 0 of the tile): lane i inspects tile j - i, 32
// predecessors per step; the nearest one with an inclusive count ends the
// walk.  Returns false if a predecessor never published (bounded spin).
__device__ bool rle_lookback(const unsigned long long *state, unsigned stride, uint64_t tile, uint64_t &excl) {
    const unsigned lane = threadIdx.x & 31u;
    excl = 0;
    for (int64_t j = int64_t(tile) - 1; j >= 0; j -= 32) {
        const int64_t me = j - int64_t(lane);
        unsigned long long r = kRleFlagInc;  // lanes before tile 0 act as an empty inclusive prefix
        if (me >= 0) {
            for (unsigned spins = 0; spins < kSpinLimit; spins++) {
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(r) : "l"(state + me * stride) : "memory");
                if (r & 3u) break;
            }
        }
        const unsigned f = unsigned(r & 3u);
        if (__any_sync(0xFFFFFFFFu, f == 0)) return false;
        const unsigned inc = __ballot_sync(0xFFFFFFFFu, f == kRleFlagInc);
        const unsigned stop = inc ? unsigned(__ffs(inc) - 1) : 32u;  // lanes 0..stop count
        uint64_t s = lane <= stop ? r >> 2 : 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, d);
        excl += s;
        if (inc) break;
    }
    return true;
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

constexpr unsigned kRleThreads = 256;
constexpr unsigned kRleRunsPerThread = 8;
constexpr unsigned kRleTile = kRleThreads * kRleRunsPerThread;  // most runs per decoder tile
constexpr unsigned kRleRows = 8192;  // output rows per decoder CTA
// Runs per decoder tile: about as many as one output chunk of kRleRows rows
// holds at the column's mean run length, a power of two in [kRleThreads,
// kRleTile].  Long runs thus mean small tiles, so a chunk loads and scans
// few runs it does not write.
inline unsigned rle_tile_runs(uint64_t n, uint64_t runs) {
    unsigned tr = kRleTile;
    while (tr > kRleThreads && uint64_t(tr) * n > uint64_t(kRleRows) * runs) tr >>= 1;
    return tr;
}

// Decoder, pass 1: run lengths summed per tile of kRleTile runs.
__global__ void __launch_bounds__(kRleThreads) k_rle_tile_rows(const uint64_t *__restrict__ pairs, uint64_t runs,
                                                              unsigned tr, uint64_t *__restrict__ tile_rows) {
    __shared__ uint64_t s_w[kRleThreads / 32];
    const uint64_t t = blockIdx.x, base = t * tr;
    uint64_t s = 0;
    for (unsigned i = threadIdx.x; i < tr; i += kRleThreads) {
        const uint64_t r = base + i;
        if (r < runs) s += __ldg(pairs + 2 * r + 1);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, d);
    if ((threadIdx.x & 31u) == 0) s_w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint64_t tot = 0;
        for (unsigned w = 0; w < kRleThreads / 32; w++) tot += s_w[w];
        tile_rows[t] = tot;
    }
}

// Decoder, pass 2: the run tile holding the first row of every chunk of
// kRleRows output rows (one thread per chunk, binary search over the tiles'
// first rows).

__global__ void k_rle_chunk_tiles(const uint64_t *__restrict__ tile_first, uint64_t ntiles, uint64_t chunks,
                                  uint32_t *__restrict__ chunk_tile) {
    for (uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < chunks; c += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t row0 = c * kRleRows;
        uint64_t lo = 0, hi = ntiles;  // last tile whose first row <= row0
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) / 2;
            if (tile_first[mid] <= row0) lo = mid;
            else hi = mid;
        }
        chunk_tile[c] = uint32_t(lo);
    }
}

// Decoder, pass 3: each CTA writes kRleRows output rows.  Starting at the
// run tile that holds its first row, it stages that tile's pairs in shared
// memory and turns them into (value, start) lists -- zero-length runs
// dropped, as they write nothing (rle.h:238-249) -- while marking each run
// start inside its rows in a bitmap (one 32-bit word per 32 rows).  Each
// warp then writes a contiguous range of words: row 32 u + l belongs to the
// run counted by the starts before word u plus the bits of word u at or
// below l.  It moves on to the next tile until its rows are done.  RPT runs
// per thread: the tile holds RPT * kRleThreads runs.
template <unsigned RPT>
__global__ void __launch_bounds__(kRleThreads) k_rle_expand(const uint64_t *__restrict__ pairs, uint64_t runs,
                                                           const uint64_t *__restrict__ tile_first, uint64_t ntiles,
                                                           const uint32_t *__restrict__ chunk_tile,
                                                           const uint64_t *__restrict__ total_rows, uint64_t n,
                                                           uint64_t *__restrict__ out, unsigned *err) {
    constexpr unsigned NWP = kRleThreads / 32, TR = RPT * kRleThreads, NWD = kRleRows / 32;
    __shared__ uint64_t s_val[TR];
    __shared__ uint64_t s_len[TR];  // lengths, then (as 32-bit words) the kept runs' entries
    __shared__ unsigned s_bits[NWD];  // run starts per 32-row word of the CTA's rows
    __shared__ uint64_t s_wsum[NWP];
    __shared__ unsigned s_wcnt[NWP];
    // a kept run's entry is 1 + its start's offset from row0 (0: it starts
    // before row0): row row0 + r lies in the last run whose entry is <= r + 1
    uint32_t *const s_st = reinterpret_cast<uint32_t *>(s_len);
    const uint64_t row0 = uint64_t(blockIdx.x) * kRleRows;
    if (row0 >= n) return;
    const uint64_t row1 = minu(n, row0 + kRleRows);
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const unsigned incl = (2u << lane) - 1u;  // lanes 0..lane
    for (uint64_t t = chunk_tile[blockIdx.x]; t < ntiles && tile_first[t] < row1; t++) {
        const uint64_t rbase = t * TR;
        const unsigned nr = unsigned(minu(TR, runs - rbase));
        // the tile's pairs into shared memory, one 16-byte pair per thread and step
#pragma unroll
        for (unsigned k = 0; k < RPT; k++) {
            const unsigned j = threadIdx.x + k * kRleThreads;
            const ulonglong2 pr = j < nr ? __ldg(reinterpret_cast<const ulonglong2 *>(pairs) + rbase + j)
                                         : make_ulonglong2(0, 0);
            s_val[j] = pr.x;
            s_len[j] = pr.y;
        }
        for (unsigned w = threadIdx.x; w < NWD; w += kRleThreads) s_bits[w] = 0;
        __syncthreads();
        // this thread's RPT consecutive runs: exclusive scans of the lengths
        // and of the number of non-empty runs
        const unsigned j0 = threadIdx.x * RPT;
        uint64_t len[RPT], val[RPT], sum = 0;
        unsigned cnt = 0;
#pragma unroll
        for (unsigned k = 0; k < RPT; k++) {
            len[k] = s_len[j0 + k];
            val[k] = s_val[j0 + k];
            sum += len[k];
            cnt += len[k] != 0;
        }
        uint64_t isum = sum;
        unsigned icnt = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t o = __shfl_up_sync(0xFFFFFFFFu, isum, d);
            const unsigned co = __shfl_up_sync(0xFFFFFFFFu, icnt, d);
            if (int(lane) >= d) {
                isum += o;
                icnt += co;
            }
        }
        if (lane == 31) {
            s_wsum[wid] = isum;
            s_wcnt[wid] = icnt;
        }
        __syncthreads();
        // the warps before this one: lanes 0..NWP-1 scan the warp totals
        uint64_t ws = lane < NWP ? s_wsum[lane] : 0;
        unsigned wc = lane < NWP ? s_wcnt[lane] : 0;
#pragma unroll
        for (int d = 1; d < int(NWP); d <<= 1) {
            const uint64_t o = __shfl_up_sync(0xFFFFFFFFu, ws, d);
            const unsigned co = __shfl_up_sync(0xFFFFFFFFu, wc, d);
            if (int(lane) >= d) {
                ws += o;
                wc += co;
            }
        }
        const unsigned kept = __shfl_sync(0xFFFFFFFFu, wc, NWP - 1);
        const uint64_t wpre = wid ? __shfl_sync(0xFFFFFFFFu, ws, wid - 1) : 0;
        const unsigned cpre = wid ? __shfl_sync(0xFFFFFFFFu, wc, wid - 1) : 0;
        uint64_t run = tile_first[t] + wpre + isum - sum;
        unsigned pos = cpre + icnt - cnt;
#pragma unroll
        for (unsigned k = 0; k < RPT; k++) {
            if (len[k]) {
                const uint32_t e = run < row0 ? 0u : uint32_t(minu(run - row0 + 1, 0xFFFFFFFFull));
                s_st[pos] = e;
                s_val[pos] = val[k];
                if (e - 1u < kRleRows) atomicOr(&s_bits[(e - 1u) >> 5], 1u << ((e - 1u) & 31u));
                pos++;
            }
            run += len[k];
        }
        __syncthreads();
        const uint64_t tile_end = t + 1 < ntiles ? tile_first[t + 1] : n;
        const uint64_t a = maxu(row0, tile_first[t]), b = minu(row1, tile_end);
        if (a < b) {
            const uint32_t ra = uint32_t(a - row0), rb = uint32_t(b - row0);
            const uint32_t tw0 = ra >> 5, tw1 = (rb + 31) >> 5;
            // the words split evenly over the warps
            const uint32_t per = (tw1 - tw0 + NWP - 1) / NWP;
            const uint32_t u0 = tw0 + wid * per, u1 = min(tw1, u0 + per);
            if (u0 < u1) {
                unsigned lo = 0, hi = kept;  // runs with entry <= 32 u0
                while (lo < hi) {
                    const unsigned mid = (lo + hi) >> 1;
                    if (s_st[mid] > 32 * u0) hi = mid;
                    else lo = mid + 1;
                }
                unsigned before = lo - 1u;  // index of the run holding row 32 u0 - 1 (wraps for none)
                uint64_t *const o = out + row0 + lane;
                for (uint32_t u = u0; u < u1; u++) {
                    const unsigned bits = s_bits[u];
                    const uint32_t r = 32 * u + lane;
                    if (r >= ra && r < rb) o[32 * u] = s_val[min(before + __popc(bits & incl), kept - 1)];
                    before += __popc(bits);
                }
            }
        }
        __syncthreads();
    }
    // the run lengths must add up to the column's length
    if (blockIdx.x == 0 && threadIdx.x == 0 && *total_rows != n) atomicOr(err, kErrCorrupt);
}

// One-pass decoder for short runs (mean length <= kRleLbMaxMean): a CTA takes
// the next tile of kRleLbTile runs from a ticket counter, stages its pairs in
// shared memory (cp.async), scans the lengths, compacts the non-empty runs to
// (value, start within the tile), publishes the tile's row count and finds the
// rows before it by the same decoupled look-back as the encoder (warp 0),
// then writes the tile's rows in windows of kRleLbWin rows through per-32-row
// bitmaps of run starts.  Each pair is read once (the two-pass decoder reads
// every pair twice, which for runs of one row is 32 B read per 8 B written).
// Shared-memory pairs sit at slot i + i / 8, so that the threads' runs
// (eight consecutive per thread) fall in different banks.  Writes stop at row
// n whatever the lengths say; lengths that do not add up to n are reported by
// the last tile (kErrCorrupt).  Needs 16-byte aligned pairs.
constexpr unsigned kRleLbThreads = 512, kRleLbRpt = 8;
constexpr unsigned kRleLbTile = kRleLbThreads * kRleLbRpt;  // runs per tile
constexpr unsigned kRleLbWin = 8192;                        // rows per write window
constexpr uint64_t kRleLbMaxMean = 4;
__host__ __device__ constexpr unsigned rle_lb_slot(unsigned i) { return i + (i >> 3); }

__global__ void __launch_bounds__(kRleLbThreads, 2) k_rle_expand_lb(const uint64_t *__restrict__ pairs,
                                                                   uint64_t runs, uint64_t n, unsigned long long *state,
                                                                   unsigned stride, unsigned *ticket,
                                                                   uint64_t *__restrict__ out, unsigned *err) {
    constexpr unsigned NW = kRleLbThreads / 32, NWD = kRleLbWin / 32;
    extern __shared__ __align__(128) uint8_t rle_smem[];
    // the tile's pairs, then (value, start within the tile) of its non-empty runs
    ulonglong2 *const s_p = reinterpret_cast<ulonglong2 *>(rle_smem);
    __shared__ unsigned s_bits[NWD];
    __shared__ uint64_t s_wsum[NW];
    __shared__ unsigned s_wcnt[NW];
    __shared__ uint64_t s_tile, s_base;
    const unsigned lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const unsigned incl = (2u << lane) - 1u;  // lanes 0..lane
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    const uint64_t ntiles = (runs + kRleLbTile - 1) / kRleLbTile;
    if (tile >= ntiles) return;
    const uint64_t rb = tile * kRleLbTile;
    const unsigned nr = unsigned(minu(kRleLbTile, runs - rb));
    for (unsigned q = threadIdx.x; q < nr; q += kRleLbThreads) cp_async16(s_p + rle_lb_slot(q), pairs + 2 * (rb + q));
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // this thread's kRleLbRpt consecutive runs: scans of lengths and of non-empty runs
    const unsigned j0 = threadIdx.x * kRleLbRpt;
    uint64_t len[kRleLbRpt], val[kRleLbRpt], sum = 0;
    unsigned cnt = 0;
#pragma unroll
    for (unsigned k = 0; k < kRleLbRpt; k++) {
        const ulonglong2 pr = j0 + k < nr ? s_p[rle_lb_slot(j0 + k)] : make_ulonglong2(0, 0);
        val[k] = pr.x;
        len[k] = pr.y;
        sum += len[k];
        cnt += len[k] != 0;
    }
    uint64_t isum = sum;
    unsigned icnt = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t o = __shfl_up_sync(0xFFFFFFFFu, isum, d);
        const unsigned co = __shfl_up_sync(0xFFFFFFFFu, icnt, d);
        if (int(lane) >= d) {
            isum += o;
            icnt += co;
        }
    }
    if (lane == 31) {
        s_wsum[wid] = isum;
        s_wcnt[wid] = icnt;
    }
    __syncthreads();  // every thread has its pairs in registers: s_p may be overwritten
    uint64_t ws = lane < NW ? s_wsum[lane] : 0;
    unsigned wc = lane < NW ? s_wcnt[lane] : 0;
#pragma unroll
    for (int d = 1; d < int(NW); d <<= 1) {
        const uint64_t o = __shfl_up_sync(0xFFFFFFFFu, ws, d);
        const unsigned co = __shfl_up_sync(0xFFFFFFFFu, wc, d);
        if (int(lane) >= d) {
            ws += o;
            wc += co;
        }
    }
    const uint64_t agg = __shfl_sync(0xFFFFFFFFu, ws, NW - 1);  // the tile's rows
    const unsigned kept = __shfl_sync(0xFFFFFFFFu, wc, NW - 1);
    const uint64_t st0 = (wid ? __shfl_sync(0xFFFFFFFFu, ws, wid - 1) : 0) + isum - sum;  // my first run's start
    {
        unsigned pos = (wid ? __shfl_sync(0xFFFFFFFFu, wc, wid - 1) : 0) + icnt - cnt;
        uint64_t run = st0;
#pragma unroll
        for (unsigned k = 0; k < kRleLbRpt; k++) {
            if (len[k]) s_p[rle_lb_slot(pos++)] = make_ulonglong2(val[k], run);
            run += len[k];
        }
    }
    // publish the tile's rows, then the rows before it
    unsigned long long *me = state + tile * stride;
    if (threadIdx.x == 0 && tile > 0) rle_publish(me, kRleFlagAgg, agg);
    if (wid == 0) {
        uint64_t excl = 0;
        if (tile > 0 && !rle_lookback(state, stride, tile, excl) && lane == 0) atomicOr(err, kErrTimeout);
        if (lane == 0) {
            rle_publish(me, kRleFlagInc, excl + agg);
            s_base = excl;
            if (tile == ntiles - 1 && excl + agg != n) atomicOr(err, kErrCorrupt);
        }
    }
    __syncthreads();
    const uint64_t base = s_base;
    if (base >= n) return;
    const uint64_t rows = minu(agg, n - base);  // never past row n
    for (uint64_t w0 = 0; w0 < rows; w0 += kRleLbWin) {
        for (unsigned w = threadIdx.x; w < NWD; w += kRleLbThreads) s_bits[w] = 0;
        __syncthreads();
        {
            // this thread's run starts in the window, one OR per bitmap word
            uint64_t s = st0;
            unsigned cw = ~0u, acc = 0;
#pragma unroll
            for (unsigned k = 0; k < kRleLbRpt; k++) {
                const uint64_t o = s - w0;  // start within the window (wraps when before it)
                if (len[k] && o < kRleLbWin) {
                    const unsigned wi = unsigned(o >> 5);
                    if (wi != cw) {
                        if (acc) atomicOr(&s_bits[cw], acc);
                        cw = wi;
                        acc = 0;
                    }
                    acc |= 1u << (o & 31u);
                }
                s += len[k];
            }
            if (acc) atomicOr(&s_bits[cw], acc);
        }
        __syncthreads();
        const unsigned wr = unsigned(minu(kRleLbWin, rows - w0));
        const unsigned nwd = (wr + 31) / 32, per = (nwd + NW - 1) / NW;
        const unsigned u0 = wid * per, u1 = min(nwd, u0 + per);
        if (u0 < u1) {
            unsigned lo = 0, hi = kept;  // runs starting before the warp's first row
            const uint64_t r0 = w0 + 32ull * u0;
            while (lo < hi) {
                const unsigned mid = (lo + hi) >> 1;
                if (s_p[rle_lb_slot(mid)].y < r0) lo = mid + 1;
                else hi = mid;
            }
            unsigned before = lo - 1u;  // index of the run holding the row before (wraps for none)
            uint64_t *const o = out + base + w0 + lane;
            for (unsigned u = u0; u < u1; u++) {
                const unsigned bits = s_bits[u];
                if (32 * u + lane < wr) o[32 * u] = s_p[rle_lb_slot(min(before + __popc(bits & incl), kept - 1))].x;
                before += __popc(bits);
            }
        }
        __syncthreads();
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
namespace {

// Driver functions for the partition of the device that a launch runs on.
struct Partition {
    CUresult (*current)(CUcontext *) = nullptr;
    CUresult (*of_ctx)(CUcontext, CUdevResource *, CUdevResourceType) = nullptr;
    CUresult (*green)(CUstream, CUgreenCtx *) = nullptr;
    CUresult (*of_green)(CUgreenCtx, CUdevResource *, CUdevResourceType) = nullptr;
    Partition() {
        get("cuCtxGetCurrent", current);
        get("cuCtxGetDevResource", of_ctx);
        get("cuStreamGetGreenCtx", green);
        get("cuGreenCtxGetDevResource", of_green);
    }
    template <class F> static void get(const char *name, F &f) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            f = reinterpret_cast<F>(p);
    }
};

}  // namespace

// SMs that a launch on `st` gets: those of the stream's or the current green
// context, else all.
static unsigned launch_sms(cudaStream_t st) {
    static const Partition d;
    unsigned sms = unsigned(sm_count());
    CUdevResource r;
    CUcontext ctx = nullptr;
    if (d.current && d.of_ctx && d.current(&ctx) == CUDA_SUCCESS && ctx &&
        d.of_ctx(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
        sms = unsigned(minu(sms, r.sm.smCount));
    CUgreenCtx g = nullptr;
    const bool own = st && st != cudaStreamLegacy && st != cudaStreamPerThread;
    if (own && d.green && d.of_green && d.green(st, &g) == CUDA_SUCCESS && g &&
        d.of_green(g, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
        sms = unsigned(minu(sms, r.sm.smCount));
    return unsigned(maxu(sms, 1));
}

// Launch of a rounds kernel: one CTA per SM at most, all resident (the kernels
// take any number of CTAs).
template <class... P, class... A>
static int launch_rounds(void (*kern)(P...), uint64_t ntiles, cudaStream_t st, A... args) {
    constexpr size_t smem = kRdSmem;
    MS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.gridDim = dim3(unsigned(minu(ntiles, launch_sms(st))));
    lc.blockDim = dim3(kRdThreads);
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    lc.attrs = at;
    lc.numAttrs = 1;
    MS_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, P(args)...));
    return MS_OK;
}

static int encode_rle(const uint64_t *d_in, uint64_t n, ms_col *out, ms_arena *a, cudaStream_t st) {
    const uint64_t tiles = (n + kRdRows - 1) / kRdRows;
    uint8_t *data = arena_take_t<uint8_t>(a, 16 * n + 64);
    // a line per word if there is room, else side by side; and the number of runs
    uint64_t nwords = tiles * kRdWordStride;
    unsigned *words = arena_take_t<unsigned>(a, nwords + 2);
    const bool lines = words;
    if (!lines) words = arena_take_t<unsigned>(a, (nwords = (tiles + 1) / 2 * 2) + 2);
    if (!data || !words) return ms_fail(MS_ERR_NOMEM, "arena exhausted (rle)");
    uint64_t runs = 0;
    if (n) {
        uint64_t *d_runs = reinterpret_cast<uint64_t *>(words + nwords);
        MS_CUDA_TRY(cudaMemsetAsync(words, 0, 4 * (nwords + 2), st));
        int rc = launch_rounds(lines ? k_rle_encode<kRdWordStride> : k_rle_encode<1>, tiles, st, d_in, n, words,
                               (ulonglong2 *)data, d_runs, a->d_err);
        if (rc) return rc;
        ReadBack back(a, st);
        const uint64_t *h_runs = back.add(d_runs);
        rc = back.wait();  // synchronises the stream
        if (rc) return rc;
        runs = *h_runs;
    }
    *out = ms_col{};
    out->format = MS_FMT_RLE;
    out->count_values = n;
    out->size_used_byte = 16 * runs;
    out->size_compr_byte = 16 * runs;
    out->size_alloc_byte = 16 * n + 64;
    out->data = data;
    return MS_OK;
}

static int decode_rle(const ms_col *in, uint64_t *d_out, ms_arena *a, cudaStream_t st) {
    const uint64_t runs = in->size_used_byte / 16, n = in->count_values;
    if (!n) return MS_OK;
    if (!runs) return ms_fail(MS_ERR_CORRUPT, "rle column with values but no runs");
    if (n <= kRleLbMaxMean * runs && (reinterpret_cast<uintptr_t>(in->data) & 15u) == 0) {
        // short runs: one pass with a look-back
        const uint64_t tiles = (runs + kRleLbTile - 1) / kRleLbTile;
        unsigned *ticket = arena_take_t<unsigned>(a, 2);
        // a line per state if there is room, else side by side
        unsigned stride = kRleStateStride;
        unsigned long long *state = arena_take_t<unsigned long long>(a, tiles * stride);
        if (!state) state = arena_take_t<unsigned long long>(a, tiles * (stride = 1));
        if (!state || !ticket) return ms_fail(MS_ERR_NOMEM, "arena exhausted (rle decode)");
        MS_CUDA_TRY(cudaMemsetAsync(state, 0, 8 * tiles * stride, st));
        MS_CUDA_TRY(cudaMemsetAsync(ticket, 0, sizeof(unsigned), st));
        constexpr size_t smem = size_t(rle_lb_slot(kRleLbTile)) * 16;
        MS_CUDA_TRY(cudaFuncSetAttribute(k_rle_expand_lb, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        k_rle_expand_lb<<<unsigned(tiles), kRleLbThreads, smem, st>>>((const uint64_t *)in->data, runs, n, state, stride,
                                                                      ticket, d_out, a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
        return MS_OK;
    }
    const unsigned tr = rle_tile_runs(n, runs);
    const uint64_t tiles = (runs + tr - 1) / tr;
    uint64_t *trows = arena_take_t<uint64_t>(a, tiles + 1);
    uint64_t *tfirst = arena_take_t<uint64_t>(a, tiles + 1);
    uint64_t *tot = arena_take_t<uint64_t>(a, 1);
    uint64_t *scr = arena_take_t<uint64_t>(a, scan_scratch_words(tiles));
    if (!trows || !tfirst || !tot || !scr) return ms_fail(MS_ERR_NOMEM, "arena exhausted (rle decode)");
    const uint64_t *pairs = (const uint64_t *)in->data;
    k_rle_tile_rows<<<unsigned(tiles), kRleThreads, 0, st>>>(pairs, runs, tr, trows);
    MS_CUDA_TRY(cudaGetLastError());
    MS_CUDA_TRY(scan_exclusive<uint64_t>(trows, tiles, tfirst, tot, scr, st));
    const uint64_t chunks = (n + kRleRows - 1) / kRleRows;
    uint32_t *ctile = arena_take_t<uint32_t>(a, chunks + 1);
    if (!ctile) return ms_fail(MS_ERR_NOMEM, "arena exhausted (rle decode)");
    k_rle_chunk_tiles<<<unsigned(minu((chunks + 255) / 256, uint64_t(persistent_grid(256, 4)))), 256, 0, st>>>(
        tfirst, tiles, chunks, ctile);
    MS_CUDA_TRY(cudaGetLastError());
    switch (tr / kRleThreads) {
    case 1: k_rle_expand<1><<<unsigned(chunks), kRleThreads, 0, st>>>(pairs, runs, tfirst, tiles, ctile, tot, n, d_out, a->d_err); break;
    case 2: k_rle_expand<2><<<unsigned(chunks), kRleThreads, 0, st>>>(pairs, runs, tfirst, tiles, ctile, tot, n, d_out, a->d_err); break;
    case 4: k_rle_expand<4><<<unsigned(chunks), kRleThreads, 0, st>>>(pairs, runs, tfirst, tiles, ctile, tot, n, d_out, a->d_err); break;
    default: k_rle_expand<8><<<unsigned(chunks), kRleThreads, 0, st>>>(pairs, runs, tfirst, tiles, ctile, tot, n, d_out, a->d_err); break;
    }
    MS_CUDA_TRY(cudaGetLastError());
    return MS_OK;
}

// Shared encoder: `ncompr` rows (a block multiple) go to the compressed part
// with page layout L, rows [ncompr, n) to the uncompressed rest.
static int encode(const uint64_t *d_in, uint64_t n, uint64_t ncompr, Layout L, ms_col *out, ms_arena *a,
                  cudaStream_t st) {
    const int fmt = L.fmt;
    const uint64_t nb = ncompr / kBlock, nrest = n - ncompr;
    const uint64_t cap = ms_size_max_byte_any_len(fmt, L.bw, n);
    uint8_t *data = arena_take_t<uint8_t>(a, cap);
    if (!data) return ms_fail(MS_ERR_NOMEM, "arena exhausted (encode)");
    uint64_t *index = nullptr, *refs = nullptr, *d_compr = nullptr;
    const unsigned grid = persistent_grid(256, 8);
    uint64_t compr = 0;
    if (nb && fmt == MS_FMT_STATIC_VBP) {
        compr = nb * 64ull * L.bw;
        k_pack_static<<<grid, 256, 0, st>>>(d_in, nb, L.bw, data, a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
    } else if (nb) {
        const uint64_t ntiles = (nb + kEncBlocks - 1) / kEncBlocks, nwords = ntiles * kRdWordStride;
        index = arena_take_t<uint64_t>(a, nb + 1);
        if (fmt == MS_FMT_FOR_DVBP) refs = arena_take_t<uint64_t>(a, nb / 2 + 1);
        unsigned *words = arena_take_t<unsigned>(a, nwords + 2);  // and the compressed size
        if (!index || !words || (fmt == MS_FMT_FOR_DVBP && !refs)) return ms_fail(MS_ERR_NOMEM, "arena exhausted (encode scratch)");
        d_compr = reinterpret_cast<uint64_t *>(words + nwords);
        MS_CUDA_TRY(cudaMemsetAsync(words, 0, 4 * (nwords + 2), st));
        auto kern = fmt == MS_FMT_DYNAMIC_VBP ? k_encode<MS_FMT_DYNAMIC_VBP>
                    : fmt == MS_FMT_DELTA_DVBP ? k_encode<MS_FMT_DELTA_DVBP> : k_encode<MS_FMT_FOR_DVBP>;
        int rc = launch_rounds(kern, ntiles, st, d_in, nb, L, words, data, index, refs, nrest, d_compr, a->d_err);
        if (rc) return rc;
        if (fmt == MS_FMT_DYNAMIC_VBP && L.dvbp_shift > 2) {
            const unsigned page = 1u << L.dvbp_shift;
            const uint64_t bytes = (nb + page - 1) / page * kPageBlocks;
            k_headers_dvbp<<<unsigned(minu((bytes + 255) / 256, grid)), 256, 0, st>>>(nb, page, index, data);
            MS_CUDA_TRY(cudaGetLastError());
        }
        if (fmt == MS_FMT_FOR_DVBP && L.for_shift > 1) {
            const unsigned page = 1u << L.for_shift;
            const uint64_t hw = (nb / 2 + page - 1) / page * 8;
            k_headers_for<<<unsigned(minu((hw + 255) / 256, grid)), 256, 0, st>>>(nb / 2, page, index, refs, data);
            MS_CUDA_TRY(cudaGetLastError());
        }
    }
    if (nrest && (!d_compr || nrest > kEncRest)) {
        k_copy_rest<<<(unsigned)minu((nrest + 255) / 256, 1024), 256, 0, st>>>(d_in + ncompr, nrest, fmt, L.bw, d_compr,
                                                                               compr, data);
        MS_CUDA_TRY(cudaGetLastError());
    }
    ReadBack back(a, st);
    const uint64_t *h_compr = d_compr ? back.add(d_compr) : &compr;
    int rc = back.wait();  // synchronises
    if (rc) return rc;
    compr = *h_compr;
    *out = ms_col{};
    out->format = uint32_t(fmt);
    out->bw = fmt == MS_FMT_STATIC_VBP ? L.bw : 0;
    out->count_values = n;
    out->size_compr_byte = compr;
    out->size_used_byte = nrest ? rest_offset(fmt, L.bw, compr) + 8 * nrest : compr;
    out->size_alloc_byte = cap;
    out->data = data;
    out->index = index;
    out->index_aux = refs;
    out->n_index = index ? nb : 0;
    return MS_OK;
}

int compress_values(const uint64_t *d_in, uint64_t n, int fmt, unsigned bw, ms_col *out, ms_arena *a,
                    cudaStream_t st) {
    if (fmt == MS_FMT_RLE) return encode_rle(d_in, n, out, a, st);
    if (fmt == MS_FMT_UNCOMPR) {
        uint64_t *data = arena_take_t<uint64_t>(a, n + 1);
        if (!data) return ms_fail(MS_ERR_NOMEM, "arena exhausted (copy)");
        if (n) MS_CUDA_TRY(cudaMemcpyAsync(data, d_in, 8 * n, cudaMemcpyDeviceToDevice, st));
        *out = ms_col{};
        out->format = MS_FMT_UNCOMPR;
        out->count_values = n;
        out->size_used_byte = 8 * n;
        out->size_alloc_byte = 8 * n;
        out->data = data;
        return MS_OK;
    }
    if (fmt == MS_FMT_STATIC_VBP && (bw < 1 || bw > 64)) return ms_fail(MS_ERR_INVALID, "static_vbp bw must be 1..64");
    if (fmt < 0 || fmt > MS_FMT_RLE) return ms_fail(MS_ERR_INVALID, "unknown format");
    const uint64_t b = block_size(fmt);
    Layout L{fmt, bw, 6, 3};  // 64 blocks, 8 cascade blocks a page
    return encode(d_in, n, n / b * b, L, out, a, st);
}

int write_values(const uint64_t *d_vals, uint64_t n_vec, uint64_t n_scalar, int fmt, unsigned bw, ms_col *out,
                 ms_arena *a, cudaStream_t st) {
    const uint64_t n = n_vec + n_scalar;
    if (fmt == MS_FMT_UNCOMPR) {
        // uncompr write iterator: the values as they are (uncompr.h:126-237)
        *out = ms_col{};
        out->format = MS_FMT_UNCOMPR;
        out->count_values = n;
        out->size_used_byte = 8 * n;
        out->size_alloc_byte = 8 * n;
        out->data = const_cast<uint64_t *>(d_vals);
        return MS_OK;
    }
    if (fmt == MS_FMT_RLE) return ms_fail(MS_ERR_UNSUPPORTED, "rle_f has no write iterator");
    if (fmt == MS_FMT_STATIC_VBP && (bw < 1 || bw > 64)) return ms_fail(MS_ERR_INVALID, "static_vbp bw must be 1..64");
    if (fmt < 0 || fmt > MS_FMT_RLE) return ms_fail(MS_ERR_INVALID, "unknown format");
    const uint64_t b = block_size(fmt);
    const uint64_t full = n_vec / kWiBuffer * kWiBuffer;
    const uint64_t ncompr = full + (n_vec - full) / b * b;
    Layout L{fmt, bw, 2, 1};  // 2048 values a page
    return encode(d_vals, n, ncompr, L, out, a, st);
}

int decompress_to(const ms_col *in, uint64_t *d_out, ms_arena *a, cudaStream_t st) {
    if (in->format == MS_FMT_RLE) return decode_rle(in, d_out, a, st);
    ColView v;
    int rc = in->format == MS_FMT_DELTA_DVBP ? prepare_view_plain(in, a, st, &v) : prepare_view(in, a, st, &v);
    if (rc) return rc;
    if (!v.n) return MS_OK;
    const uint64_t nbt = v.nblocks_total();
    if (in->format == MS_FMT_DELTA_DVBP && v.nb()) {
        DeltaSegs segs;
        rc = delta_segments(v, in->index_aux, nullptr, nullptr, &segs, a, st);
        if (rc) return rc;
        const uint64_t units = segs.nseg + nbt - v.nb();
        k_decode_delta<<<(unsigned)minu((units + 7) / 8, persistent_grid(256, 3)), 256, 0, st>>>(v, segs, d_out,
                                                                                               a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
        return MS_OK;
    }
    const unsigned grid = (unsigned)minu((nbt + 7) / 8, persistent_grid(256, 8));
    k_decode_all<<<grid, 256, 0, st>>>(v, d_out, a->d_err);
    MS_CUDA_TRY(cudaGetLastError());
    return MS_OK;
}

}  // namespace ms

extern "C" int ms_gpu_morph(const ms_col *src, int dst_format, unsigned dst_bw, ms_col *out, ms_arena *a,
                            void *stream) {
    using namespace ms;
    if (!src || !out || !a) return ms_fail(MS_ERR_INVALID, "morph: null argument");
    int rc = check_col(src, false);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    // morph from a format to itself returns the input (morph.h:133-160)
    if (int(src->format) == dst_format && (dst_format != MS_FMT_STATIC_VBP || src->bw == dst_bw)) {
        *out = *src;
        return MS_OK;
    }
    if (src->format == MS_FMT_UNCOMPR)
        return compress_values((const uint64_t *)src->data, src->count_values, dst_format, dst_bw, out, a, st);
    // decompress (possibly followed by a compress into another format)
    uint64_t *tmp = arena_take_t<uint64_t>(a, src->count_values + 1);
    if (!tmp) return ms_fail(MS_ERR_NOMEM, "arena exhausted (morph)");
    rc = decompress_to(src, tmp, a, st);
    if (rc) return rc;
    if (dst_format == MS_FMT_UNCOMPR) {
        rc = read_err(a, st);
        if (rc) return rc;
        *out = ms_col{};
        out->format = MS_FMT_UNCOMPR;
        out->count_values = src->count_values;
        out->size_used_byte = 8 * src->count_values;
        out->size_alloc_byte = 8 * src->count_values;
        out->data = tmp;
        return MS_OK;
    }
    return compress_values(tmp, src->count_values, dst_format, dst_bw, out, a, st);
}
