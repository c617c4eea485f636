// query.cu -- the fused compressed multi-operator query:
//
//   P1 = select(filter < c)            (select_compr.h:100-260)
//   P2 = semi_join(L, fk)              (join_semi_equi_compr.h:106-300)
//   P  = intersect_sorted(P1, P2)      (intersect_compr.h:190-347)
//   G  = project(gkey, P), M = project(measure, P)
//   (gr, ext) = group(G); S = agg_sum(gr, M, |ext|)   (group_compr.h, scalar/agg_sum_uncompr.h)
//
// in one pass over the fact table: per 512-row block a warp decodes filter,
// probes fk against the build side's bitmap, and for the surviving rows
// decodes gkey and measure and folds (key, row, measure) into a per-CTA
// shared-memory group table (warp-aggregated for skewed keys), flushed to a
// global table at the end.  Each key keeps its smallest row; after a scan of
// the per-block hit counts, the group's extent -- the position of that row in
// P, which is what the reference's group operator returns -- is the hits
// before its block plus its rank within the block, and ordering groups by
// first row gives the reference's group ids.  The result equals the operator-at-a-time
// pipeline's bit for bit; no intermediate touches HBM.
#include <algorithm>
#include <vector>

#include "fastpath.cuh"
#include "internal.h"
#include "positions.cuh"
#include "scan.cuh"
#include "stream.cuh"
#include "tma.cuh"
#include "window.cuh"

namespace ms {
namespace {

constexpr unsigned kQSlots = 2048;  // per-CTA group table
constexpr uint64_t kQEmpty = ~uint64_t(0);

__device__ __forceinline__ uint64_t qhash(uint64_t k) {
    k ^= k >> 33;
    k *= 0xFF51AFD7ED558CCDull;
    k ^= k >> 33;
    return k;
}

struct GTable {  // global group table (open addressing)
    unsigned long long *keys;
    unsigned long long *first;  // smallest row of the group
    unsigned long long *sums;
    uint64_t mask;
};

// kLook: reads the slot before changing it, so that a key that is there with a
// smaller row costs two loads and one atomic instead of three atomics -- for
// rows that come one by one.  The flush of a CTA's groups meets mostly empty
// slots, or slots that other CTAs are filling, and does not look.
template <bool kLook = false>
__device__ __forceinline__ bool gtable_add(const GTable &t, uint64_t key, uint64_t first, uint64_t sum) {
    uint64_t h = qhash(key) & t.mask;
    for (uint64_t p = 0; p <= t.mask; p++) {
        unsigned long long x = kQEmpty, f = ~0ull;
        if (kLook) {
            x = ((volatile unsigned long long *)t.keys)[h];
            f = ((volatile unsigned long long *)t.first)[h];
        }
        if (x == kQEmpty) x = atomicCAS(t.keys + h, kQEmpty, key);
        if (x == kQEmpty || x == key) {
            if (first < f) atomicMin(t.first + h, first);
            atomicAdd(t.sums + h, sum);
            return true;
        }
        h = (h + 1) & t.mask;
    }
    return false;
}

// For rows beyond a CTA's table.  Out of line: inlined into the consumers' loop
// it made the pass slower, 2^27 rows that all find their group in the table
// 301 us instead of 282.
__device__ __noinline__ bool gtable_look(const GTable &t, uint64_t key, uint64_t first, uint64_t sum) {
    return gtable_add<true>(t, key, first, sum);
}

__global__ void __launch_bounds__(256) k_query3(ColView filt, ColView fk, ColView gkey, ColView meas, int cmp,
                                               uint64_t c, const uint32_t *__restrict__ bits, uint64_t lo,
                                               uint64_t span, GTable gt, uint32_t *__restrict__ blk_hits,
                                               uint64_t b_begin, unsigned *err) {
    __shared__ unsigned long long s_key[kQSlots], s_first[kQSlots], s_sum[kQSlots];
    for (unsigned i = threadIdx.x; i < kQSlots; i += blockDim.x) {
        s_key[i] = kQEmpty;
        s_first[i] = ~0ull;
        s_sum[i] = 0;
    }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    bool ok = true, fit = true;
    for (uint64_t b = b_begin + (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < filt.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16];
        unsigned valid;
        ok &= decode_block(filt, b, l, q, v, valid);
        unsigned m = select_mask(filt, b, l, q, v, valid, cmp, c);
        if (__any_sync(0xFFFFFFFFu, m != 0)) {
            unsigned vk;
            ok &= decode_block(fk, b, l, q, v, vk);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                if (!((m >> k) & 1u)) continue;
                const uint64_t d = v[k] - lo;
                const bool in = v[k] >= lo && d < span && ((bits[d >> 5] >> (d & 31u)) & 1u);
                if (!in) m &= ~(1u << k);
            }
        }
        const unsigned total = __reduce_add_sync(0xFFFFFFFFu, __popc(m));
        if (lane == 0) blk_hits[b] = total;
        if (total == 0) continue;
        uint64_t g[16], w[16];
        unsigned vg, vm;
        ok &= decode_block(gkey, b, l, q, g, vg);
        ok &= decode_block(meas, b, l, q, w, vm);
        const uint64_t row0 = b * kBlock;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const bool hit = (m >> k) & 1u;
            const uint64_t key = g[k];
            const uint64_t first = row0 + (16u * q + k) * 8u + l;
            // lanes with the same key combine first: one table update per key
            const unsigned hm = __ballot_sync(0xFFFFFFFFu, hit);
            if (!hit) continue;
            const unsigned peers = __match_any_sync(hm, key);
            uint64_t s = w[k], f = first;
            for (unsigned rest = peers; rest;) {
                const int src = __ffs(rest) - 1;
                rest &= rest - 1;
                const uint64_t so = __shfl_sync(peers, w[k], src);
                const uint64_t fo = __shfl_sync(peers, first, src);
                if (src != int(lane)) {
                    s += so;
                    f = minu(f, fo);
                }
            }
            if (int(lane) != __ffs(peers) - 1) continue;
            // per-CTA table, then the global one when the key does not fit
            uint64_t h = qhash(key) & (kQSlots - 1);
            bool done = false;
            if (key != kQEmpty) {
                for (unsigned p = 0; p < 16; p++) {
                    const unsigned long long old = atomicCAS(s_key + h, kQEmpty, key);
                    if (old == kQEmpty || old == key) {
                        atomicMin(s_first + h, (unsigned long long)f);
                        atomicAdd(s_sum + h, (unsigned long long)s);
                        done = true;
                        break;
                    }
                    h = (h + 1) & (kQSlots - 1);
                }
            }
            if (!done) fit &= gtable_add(gt, key, f, s);
        }
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < kQSlots; i += blockDim.x)
        if (s_key[i] != kQEmpty) fit &= gtable_add(gt, s_key[i], s_first[i], s_sum[i]);
    if (!ok) atomicOr(err, kErrCorrupt);
    if (!fit) atomicOr(err, kErrCapacity);
}

// ---------------------------------------------------------------------------
// Staged variant.  One persistent CTA per SM: warp 0 forms tiles of
// consecutive 512-row blocks whose bytes in all four fact columns fit one
// stage buffer and brings each column's range into shared memory with one
// bulk copy; consumer warps take the tile's blocks two at a time, round-robin.
// The filter is compared inside the bit-width switch (32 rows per thread) and
// the hits of both blocks are listed, so that their foreign keys are extracted
// and probed 128 at a time, four per lane, every lane busy; the rows that
// survive are compacted in the list, their group key and measure extracted
// together and queued per warp, and 32 queued rows at a time go to the CTA's
// group table.  The producer takes block locations from windows it loaded
// ahead (window.cuh) and forms a tile before it waits for its stage: its path
// per tile bounded the pass.  2^27 rows: 282 us (356 before; 412 with the
// listed hits alone), of which reading the columns takes 149; the rest is the
// consumers' instructions at 17 warps per SM (24 warps leave a smaller ring:
// 383 us).
// Requires the filter in uncompr/static_vbp/dynamic_vbp and the other three
// columns in those or for_f (delta_f and rows in the uncompressed rests go
// through k_query3).
// ---------------------------------------------------------------------------
constexpr unsigned kQTile = 32;  // blocks per tile (one producer lane each)
constexpr unsigned kQCols = 4;   // filter, fk, group key, measure

struct QStage {
    uint64_t b0;
    unsigned nblk;
    unsigned pad;
};

struct QCfg {
    unsigned stages;
    unsigned stage_bytes;
};

// A consumer warp's list of hits (rows of its two blocks) and queue of rows to be
// grouped (kQQueue entries: up to 31 left over and 32 new ones).
constexpr unsigned kQQueue = 64;
struct QWarp {
    unsigned long long key[kQQueue], val[kQQueue], row[kQQueue];
    uint16_t hits[2 * kBlock];  // second block << 9 | row
};

// The CTA's group table: sums as two 32-bit words (32-bit shared atomics are
// native).
struct QTable {
    unsigned long long *key, *first;
    unsigned *lo, *hi;
};

// Folds one row into the CTA's table, or into the global one when the key
// finds no place among 16 slots.  A key that is there with a smaller row
// costs two loads and one atomic.
__device__ __forceinline__ bool qtable_add(const QTable &t, const GTable &gt, uint64_t key, uint64_t row, uint64_t val) {
    if (key != kQEmpty) {
        unsigned h = unsigned(qhash(key)) & (kQSlots - 1);
        for (unsigned p = 0; p < 16; p++) {
            unsigned long long x = ((volatile unsigned long long *)t.key)[h];
            if (x == kQEmpty) x = atomicCAS(t.key + h, kQEmpty, (unsigned long long)key);
            if (x == kQEmpty || x == key) {
                if (row < ((volatile unsigned long long *)t.first)[h]) atomicMin(t.first + h, (unsigned long long)row);
                const unsigned lo = unsigned(val), old = lo ? atomicAdd(t.lo + h, lo) : 0u;
                const unsigned hi = unsigned(val >> 32) + (old + lo < old ? 1u : 0u);
                if (hi) atomicAdd(t.hi + h, hi);
                return true;
            }
            h = (h + 1) & (kQSlots - 1);
        }
    }
    return gtable_look(gt, key, row, val);
}

// value of row r (0..511) of a vbp block of width bw staged in shared memory;
// for widths up to 32 from the two 32-bit words at its first bit (the second
// one may lie up to 64 bytes behind the block, within shared memory)
__device__ __forceinline__ uint64_t vbp_extract(const uint64_t *blk, unsigned bw, unsigned r) {
    const unsigned l = r & 7u, p = (r >> 3) * bw;
    if (bw <= 32u) {
        const uint32_t *const b = reinterpret_cast<const uint32_t *>(blk) + 2u * l;
        const unsigned i = p >> 5, j = i + 1u;
        const uint32_t x = __funnelshift_r(b[(i >> 1) * 16u + (i & 1u)], b[(j >> 1) * 16u + (j & 1u)], p & 31u);
        return bw == 32u ? x : x & ((1u << bw) - 1u);
    }
    const unsigned w = p >> 6, sh = p & 63u;
    uint64_t x = blk[w * 8u + l] >> sh;
    if (sh + bw > 64u) x |= blk[(w + 1u) * 8u + l] << (64u - sh);
    return bw >= 64u ? x : x & ((uint64_t(1) << bw) - 1u);
}

__host__ __device__ inline uint64_t q3_meta_bytes(unsigned S) {
    return (uint64_t(16) * S + sizeof(QStage) * S + 5ull * kQCols * S * kQTile + 127) / 128 * 128;
}

// Where the probes read the build side's bitmap (nwords words):
enum : int {
    kBmGlobal = 0,   // global memory (an L2 round trip per probe)
    kBmShared = 1,   // the whole bitmap in this CTA's shared memory
    kBmCluster = 2,  // split over the two CTAs of a cluster: words [0, half) in
                     // rank 0, [half, nwords) in rank 1, read through
                     // distributed shared memory (ld.shared::cluster)
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// every thread of both CTAs of the cluster; shared-memory writes before it
// are visible to the other CTA after it
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ uint32_t dsmem_ld32(const uint32_t *local_base, uint32_t idx, unsigned rank) {
    uint32_t a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local_base + idx)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// kBM: where the bitmap lives (kBmGlobal / kBmShared / kBmCluster); in
// shared memory it follows the group table, so a probe costs a shared-memory
// load (local or in the partner CTA) instead of an L2 round trip.
template <int W, int kBM>
__global__ void __launch_bounds__(32 * (W + 1), 1)
    k_query3_tma(ColView fk, ColView gkey, ColView meas, StreamCol c0, StreamCol c1, StreamCol c2, StreamCol c3,
                 Pred pred, const uint32_t *__restrict__ bits, uint64_t nwords, uint64_t lo, uint64_t span, QCfg cfg,
                 GTable gt, uint32_t *__restrict__ blk_hits, unsigned *err) {
    constexpr bool kSB = kBM != kBmGlobal;
    extern __shared__ __align__(128) uint8_t smem[];
    const unsigned S = cfg.stages, SB = cfg.stage_bytes;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem);
    uint64_t *empty = full + S;
    QStage *desc = reinterpret_cast<QStage *>(empty + S);
    uint32_t *offs = reinterpret_cast<uint32_t *>(desc + S);                 // [S][kQCols][kQTile]
    uint8_t *bws = reinterpret_cast<uint8_t *>(offs + S * kQCols * kQTile);  // [S][kQCols][kQTile]
    uint8_t *ring = smem + q3_meta_bytes(S);
    QTable tab;
    tab.key = reinterpret_cast<unsigned long long *>(ring + size_t(S) * SB);
    tab.first = tab.key + kQSlots;
    tab.lo = reinterpret_cast<unsigned *>(tab.first + kQSlots);
    tab.hi = tab.lo + kQSlots;
    QWarp *const s_warp = reinterpret_cast<QWarp *>(tab.hi + kQSlots);
    uint32_t *s_bits = reinterpret_cast<uint32_t *>(s_warp + W);
    const uint32_t *pbits = kSB ? s_bits : bits;
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    for (unsigned i = threadIdx.x; i < kQSlots; i += blockDim.x) {
        tab.key[i] = kQEmpty;
        tab.first[i] = ~0ull;
        tab.lo[i] = tab.hi[i] = 0;
    }
    const uint32_t half = uint32_t((nwords + 1) / 2);  // words per CTA in a cluster
    if (kBM == kBmShared)
        for (uint64_t i = threadIdx.x; i < nwords; i += blockDim.x) s_bits[i] = __ldg(bits + i);
    if (kBM == kBmCluster) {
        const uint64_t w0 = uint64_t(cluster_rank()) * half;
        for (uint64_t i = threadIdx.x; i < half; i += blockDim.x) s_bits[i] = w0 + i < nwords ? __ldg(bits + w0 + i) : 0u;
    }
    if (threadIdx.x == 0) {
        for (unsigned st = 0; st < S; st++) {
            mbar_init(full + st, 1);
            mbar_init(empty + st, W);
        }
        mbar_fence_init();
    }
    __syncthreads();
    if (kBM == kBmCluster) cluster_sync();  // both halves of the bitmap are in place

    const uint64_t nbs = minu(minu(c0.nb, c1.nb), minu(c2.nb, c3.nb));
    const uint64_t b_lo = nbs * blockIdx.x / gridDim.x, b_hi = nbs * (blockIdx.x + 1) / gridDim.x;
    bool ok = true, fit = true, bad = false;

    if (warp == 0) {
        // ---------------- producer ----------------
        const StreamCol *const cols[kQCols] = {&c0, &c1, &c2, &c3};
        BlockWindow<kQCols> win;
        win.init(cols, b_lo, b_hi, lane);
        uint64_t b = b_lo;
        unsigned t = 0;
        for (;; t++) {
            const unsigned st = t % S, use = t / S;
            // the tile is formed before its stage is waited for
            const bool valid = b + lane < b_hi;
            uint64_t off[kQCols], x0[kQCols];
            uint32_t len[kQCols], cbase[kQCols], clen[kQCols], need = 0, acc = 0, total = 0;
            unsigned bw[kQCols];
            win.advance(cols, b, lane);
#pragma unroll
            for (unsigned c = 0; c < kQCols; c++) {
                win.get(c, b, lane, off[c], bw[c]);
                x0[c] = __shfl_sync(0xFFFFFFFFu, off[c], 0);
                len[c] = valid ? uint32_t(off[c] - x0[c]) + 64u * bw[c] : 0u;
                need += (len[c] + 127u) / 128u * 128u;
            }
            const unsigned T = __popc(__ballot_sync(0xFFFFFFFFu, valid && need <= SB));
#pragma unroll
            for (unsigned c = 0; c < kQCols; c++) {
                clen[c] = __shfl_sync(0xFFFFFFFFu, len[c], T ? T - 1 : 0);
                cbase[c] = acc;
                acc += (clen[c] + 127u) / 128u * 128u;
                total += clen[c];
            }
            // lane c brings column c
            uint64_t my_src = 0;
            uint32_t my_len = 0, my_dst = 0;
#pragma unroll
            for (unsigned c = 0; c < kQCols; c++)
                if (lane == c) {
                    my_src = reinterpret_cast<uint64_t>(cols[c]->base) + x0[c];
                    my_len = clen[c];
                    my_dst = cbase[c];
                }
            if (use > 0 && !mbar_wait(empty + st, (use - 1) & 1u)) {
                ok = false;
                break;
            }
            if (b >= b_hi || T == 0) {  // the end, or one block larger than a stage: configuration error
                if (lane == 0) {
                    if (b < b_hi) atomicOr(err, kErrCapacity);
                    desc[st].nblk = 0;
                    mbar_arrive(full + st);
                }
                ok &= b >= b_hi;
                t++;
                break;
            }
            if (lane < T) {
#pragma unroll
                for (unsigned c = 0; c < kQCols; c++) {
                    offs[(st * kQCols + c) * kQTile + lane] = st * SB + cbase[c] + uint32_t(off[c] - x0[c]);
                    bws[(st * kQCols + c) * kQTile + lane] = uint8_t(bw[c]);
                }
            }
            if (lane == 0) {
                desc[st].b0 = b;
                desc[st].nblk = T;
            }
            __threadfence_block();
            __syncwarp();
            if (lane == 0) mbar_arrive_expect_tx(full + st, total);
            __syncwarp();
            if (lane < kQCols)
                bulk_g2s(ring + st * SB + my_dst, reinterpret_cast<const uint8_t *>(my_src), my_len, full + st);
            __syncwarp();
            b += T;
        }
        const unsigned issued = t;
        for (unsigned st = 0; st < S && st < issued; st++) {
            const unsigned uses = (issued - st + S - 1) / S;
            if (!mbar_wait(full + st, (uses - 1) & 1u)) ok = false;
        }
    } else {
        // ---------------- consumers ----------------
        const unsigned cw = warp - 1, l = lane & 7u, h = (lane >> 3) & 1u, hb = lane >> 4;
        const uint64_t *const kaux = fk.fmt == MS_FMT_FOR_DVBP ? fk.aux : nullptr;
        const uint64_t *const gaux = gkey.fmt == MS_FMT_FOR_DVBP ? gkey.aux : nullptr;
        const uint64_t *const maux = meas.fmt == MS_FMT_FOR_DVBP ? meas.aux : nullptr;
        QWarp &mine = s_warp[cw];
        unsigned queued = 0;  // rows in the warp's queue
        unsigned turn = 0;    // units of the tiles before, mod W
        for (unsigned t = 0;; t++) {
            const unsigned st = t % S, use = t / S;
            if (!mbar_wait(full + st, use & 1u)) {
                ok = false;
                break;
            }
            const unsigned T = desc[st].nblk;
            if (T == 0) break;
            const uint64_t b0 = desc[st].b0;
            // One block at a time where the ring's pairs are fewer than the
            // warps: wide columns have three blocks to a tile, and with pairs
            // 6 of 16 warps worked (2^23 rows, three columns of 64 bits, 90 %
            // kept, 1000 groups: 647 us, 506 with single blocks).  Else pairs:
            // a single block's filter takes half the lanes (2^27 rows, 10 %
            // kept: 624 us a call, 532 with pairs).
            const bool two = S * ((T + 1) / 2) >= W;
            const unsigned units = two ? (T + 1) / 2 : T;
            const uint32_t *o = offs + st * kQCols * kQTile;
            const uint8_t *w = bws + st * kQCols * kQTile;
            for (unsigned u = (cw + W - turn) % W; u < units; u += W) {
                const unsigned j0 = two ? 2 * u : u, j = j0 + hb;
                unsigned m = 0;
                if (j < T && (two || !hb)) {
                    m = mask32_block_rt(w[j], reinterpret_cast<const uint64_t *>(ring + o[j]), l, h, pred, bad);
                    if (w[kQTile + j] - 1u >= 64u || w[2 * kQTile + j] - 1u >= 64u || w[3 * kQTile + j] - 1u >= 64u) {
                        bad = true;
                        m = 0;
                    }
                }
                // the hits of both blocks as a list, the first block's first
                const unsigned n = __popc(m);
                unsigned incl = n;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const unsigned x = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (int(lane) >= d) incl += x;
                }
                {
                    uint16_t *at = mine.hits + (incl - n);
                    const unsigned base = hb << 9 | h << 8 | l;
                    for (unsigned r = m; r; r &= r - 1) *at++ = uint16_t(base + 8u * unsigned(__ffs(r) - 1));
                }
                const unsigned n0 = __shfl_sync(0xFFFFFFFFu, incl, 15), hits = __shfl_sync(0xFFFFFFFFu, incl, 31);
                __syncwarp();
                unsigned alive = 0, alive0 = 0;  // surviving rows, of the first block
                for (unsigned h0 = 0; h0 < hits; h0 += 128) {
                    unsigned e[4];
                    uint32_t word[4], bit[4];
#pragma unroll
                    for (unsigned i = 0; i < 4; i++) {
                        const bool in = h0 + 32u * i + lane < hits;
                        e[i] = in ? mine.hits[h0 + 32u * i + lane] : 0u;
                        const unsigned jj = j0 + (e[i] >> 9);
                        uint64_t v = vbp_extract(reinterpret_cast<const uint64_t *>(ring + o[kQTile + jj]), w[kQTile + jj],
                                                 e[i] & 511u);
                        if (kaux) v += __ldg(kaux + ((b0 + jj) >> 1));
                        const uint64_t d = v - lo;
                        const bool inr = in && v >= lo && d < span;
                        if (kBM == kBmCluster) {
                            const uint32_t wi = uint32_t(d >> 5);
                            const unsigned own = wi >= half;
                            word[i] = inr ? dsmem_ld32(s_bits, wi - own * half, own) : 0u;
                        } else {
                            word[i] = inr ? (kSB ? pbits[d >> 5] : __ldg(pbits + (d >> 5))) : 0u;
                        }
                        bit[i] = unsigned(d & 31u);
                    }
                    __syncwarp();  // the list is in registers up to here
#pragma unroll
                    for (unsigned i = 0; i < 4; i++) {
                        const bool hit = (word[i] >> bit[i]) & 1u;
                        const unsigned hm = __ballot_sync(0xFFFFFFFFu, hit), from = h0 + 32u * i;
                        if (hit) mine.hits[alive + __popc(hm & ((1u << lane) - 1u))] = uint16_t(e[i]);
                        alive += __popc(hm);
                        alive0 += n0 >= from + 32u ? __popc(hm) : n0 > from ? __popc(hm & ((1u << (n0 - from)) - 1u)) : 0u;
                    }
                    __syncwarp();
                }
                if (lane <= unsigned(two) && j0 + lane < T) blk_hits[b0 + j0 + lane] = lane ? alive - alive0 : alive0;
                // their group keys and measures
                for (unsigned a0 = 0; a0 < alive; a0 += 32) {
                    const unsigned cnt = min(32u, alive - a0);
                    if (lane < cnt) {
                        const unsigned ee = mine.hits[a0 + lane], jj = j0 + (ee >> 9), row = ee & 511u;
                        const uint64_t blk = b0 + jj;
                        uint64_t g = vbp_extract(reinterpret_cast<const uint64_t *>(ring + o[2 * kQTile + jj]),
                                                 w[2 * kQTile + jj], row);
                        uint64_t v = vbp_extract(reinterpret_cast<const uint64_t *>(ring + o[3 * kQTile + jj]),
                                                 w[3 * kQTile + jj], row);
                        if (gaux) g += __ldg(gaux + (blk >> 1));
                        if (maux) v += __ldg(maux + (blk >> 1));
                        mine.key[queued + lane] = g;
                        mine.val[queued + lane] = v;
                        mine.row[queued + lane] = blk * kBlock + row;
                    }
                    queued += cnt;
                    __syncwarp();
                    if (queued >= 32) {
                        fit &= qtable_add(tab, gt, mine.key[lane], mine.row[lane], mine.val[lane]);
                        queued -= 32;
                        __syncwarp();
                        if (lane < queued) {
                            mine.key[lane] = mine.key[32 + lane];
                            mine.val[lane] = mine.val[32 + lane];
                            mine.row[lane] = mine.row[32 + lane];
                        }
                        __syncwarp();
                    }
                }
                __syncwarp();  // the list is free for the next pair
            }
            turn = (turn + units) % W;
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + st);
        }
        if (lane < queued) fit &= qtable_add(tab, gt, mine.key[lane], mine.row[lane], mine.val[lane]);
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < kQSlots; i += blockDim.x)
        if (tab.key[i] != kQEmpty)
            fit &= gtable_add(gt, tab.key[i], tab.first[i], ((unsigned long long)tab.hi[i] << 32) + tab.lo[i]);
    if (!ok) atomicOr(err, kErrTimeout);
    if (bad) atomicOr(err, kErrCorrupt);
    if (!fit) atomicOr(err, kErrCapacity);
    if (kBM == kBmCluster) cluster_sync();  // the partner may still read this CTA's half
}

// bitmap of the build side's keys (dense range)
__global__ void k_q3_bits(ColView l, uint64_t lo, uint32_t *bits, unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, ll = lane & 7u, q = lane >> 3;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < l.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16];
        unsigned valid;
        ok &= decode_block(l, b, ll, q, v, valid);
#pragma unroll
        for (int k = 0; k < 16; k++)
            if ((valid >> k) & 1u) {
                const uint64_t d = v[k] - lo;
                atomicOr(bits + (d >> 5), 1u << (d & 31u));
            }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
}

// Extent of every group: its first row's position in P, i.e. the hits in
// earlier blocks (scan of the per-block counts) plus the row's rank among the
// hits of its own block, which one warp per group recomputes by decoding that
// block of the filter and the foreign key again.  Results are compacted to
// dense records (key, extent, sum, first row) in arrival order.
__global__ void __launch_bounds__(256) k_q3_extents(GTable gt, ColView filt, ColView fk, int cmp, uint64_t c,
                                                   const uint32_t *__restrict__ bits, uint64_t lo, uint64_t span,
                                                   const uint64_t *__restrict__ blk_off,
                                                   unsigned long long *__restrict__ cnt,
                                                   uint64_t *__restrict__ o, unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    bool ok = true;
    // 32 slots per warp and step, the occupied ones one after another
    for (uint64_t h0 = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * 32; h0 <= gt.mask;
         h0 += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t my_key = gt.keys[h0 + lane];  // the table has a multiple of 32 slots
        for (unsigned todo = __ballot_sync(0xFFFFFFFFu, my_key != kQEmpty); todo; todo &= todo - 1) {
            const uint64_t h = h0 + unsigned(__ffs(todo) - 1);
            const uint64_t key = __shfl_sync(0xFFFFFFFFu, my_key, __ffs(todo) - 1);
            const uint64_t row = gt.first[h];
            const uint64_t b = row / kBlock;
            uint64_t v[16];
            unsigned valid;
            ok &= decode_block(filt, b, l, q, v, valid);
            unsigned m = select_mask(filt, b, l, q, v, valid, cmp, c);
            ok &= decode_block(fk, b, l, q, v, valid);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const uint64_t d = v[k] - lo;
                if (!(v[k] >= lo && d < span && ((bits[d >> 5] >> (d & 31u)) & 1u))) m &= ~(1u << k);
            }
            unsigned rank[16];
            block_ranks(m, l, q, rank);
            const unsigned s = unsigned(row % kBlock) / 8u;  // slot of the row within its lane
            unsigned rk = 0;
#pragma unroll
            for (unsigned k = 0; k < 16; k++) rk = (16u * q + k == s) ? rank[k] : rk;
            rk = __shfl_sync(0xFFFFFFFFu, rk, int((s / 16u) * 8u + unsigned(row % 8)));
            if (lane == 0) {
                const unsigned long long i = atomicAdd(cnt, 1ull);
                o[4 * i] = key;
                o[4 * i + 1] = blk_off[b] + rk;
                o[4 * i + 2] = gt.sums[h];
                o[4 * i + 3] = row;
            }
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
}

bool random_access(const ColView &v) { return plain(v) || v.fmt == MS_FMT_FOR_DVBP; }

constexpr uint64_t kQFirstGroups = 4096;  // group records read back with the counts
constexpr size_t kQSmemMax = 232448;  // 227 KiB of dynamic shared memory per CTA

// launch configuration of the staged kernel (consumer warps 8/16/24)
ms_tuning g_q3 = {1, 16, 3, 57344, 1, 16};
// device time of the last call's fact-table pass
cudaEvent_t g_q3_ev[2] = {nullptr, nullptr};
double g_q3_pass_ms = -1;

template <int W, int kBM>
int launch_q3_kern(size_t shm, QCfg cfg, const ColView &kv, const ColView &gv, const ColView &mv,
                   const StreamCol &s0, const StreamCol &s1, const StreamCol &s2, const StreamCol &s3, const Pred &pred,
                   const uint32_t *bits, uint64_t nwords, uint64_t lo, uint64_t span, const GTable &gt, uint32_t *hits,
                   unsigned *d_err, cudaStream_t st) {
    auto kern = k_query3_tma<W, kBM>;
    MS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(shm)));
    if (kBM != kBmCluster) {
        kern<<<unsigned(sm_count()), 32 * (W + 1), shm, st>>>(kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span,
                                                              cfg, gt, hits, d_err);
        MS_CUDA_TRY(cudaGetLastError());
        return MS_OK;
    }
    // clusters of two CTAs (one per SM), as many as fit at once
    cudaLaunchConfig_t lc = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.blockDim = dim3(32 * (W + 1));
    lc.dynamicSmemBytes = shm;
    lc.stream = st;
    lc.attrs = at;
    lc.numAttrs = 1;
    lc.gridDim = dim3(unsigned(sm_count() / 2 * 2));
    int ncl = 0;
    MS_CUDA_TRY(cudaOccupancyMaxActiveClusters(&ncl, kern, &lc));
    lc.gridDim = dim3(unsigned(2 * (ncl > 0 ? ncl : 1)));
    MS_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, cfg, gt, hits,
                                   d_err));
    return MS_OK;
}

template <int W>
int launch_q3_tma_w(const ColView &kv, const ColView &gv, const ColView &mv, const StreamCol &s0, const StreamCol &s1,
                    const StreamCol &s2, const StreamCol &s3, const Pred &pred, const uint32_t *bits, uint64_t nwords,
                    uint64_t lo, uint64_t span, const GTable &gt, uint32_t *hits, unsigned *d_err, cudaStream_t st) {
    QCfg cfg{g_q3.stages, g_q3.stage_bytes};
    const size_t table = 3ull * 8 * kQSlots + W * sizeof(QWarp), bitmap = 4 * nwords, half = 4 * ((nwords + 1) / 2);
    // The ring takes what the table, the warps' lists and a bitmap in shared
    // memory leave: the configured stages, shrunk to at least 24 KiB each, or
    // fewer of them (a stage holds at least one block of all columns, 16 KiB).
    // staged 1: the bitmap in shared memory beside the configured ring when
    // it fits, else in global memory.  staged 3: split over a 2-CTA cluster.
    // Both ways of making room for a large bitmap were measured slower than
    // reading it from global memory (before hits were listed, 2^20 keys, 2^26
    // fact rows): a 2 x 25 KiB ring with the whole bitmap lost more to the
    // shallower pipeline than the probes gained, and the cluster split took
    // 242 us against 198 us.
    const auto fit_ring = [&](size_t words_bytes, unsigned want) -> QCfg {
        QCfg c = cfg;
        for (;; c.stages--) {
            const size_t fixed = q3_meta_bytes(c.stages) + table + words_bytes;
            if (fixed + 2 * 16384 > kQSmemMax) return QCfg{0, 0};
            const size_t sb = minu(cfg.stage_bytes, (kQSmemMax - fixed) / c.stages / 128 * 128);
            if (sb >= minu(want, cfg.stage_bytes)) {
                c.stage_bytes = unsigned(sb);
                return c;
            }
            if (c.stages == 2) return QCfg{0, 0};
        }
    };
    int mode = kBmGlobal;
    const QCfg rs = fit_ring(bitmap, 40960), rc3 = fit_ring(half, 24576);
    if (g_q3.staged == 1 && rs.stages == cfg.stages) mode = kBmShared;
    else if (g_q3.staged == 3 && rc3.stages == cfg.stages) mode = kBmCluster;
    cfg = mode == kBmShared ? rs : mode == kBmCluster ? rc3 : fit_ring(0, 24576);
    if (!cfg.stages) return ms_fail(MS_ERR_INVALID, "query3: launch configuration does not fit shared memory");
    const size_t shm = q3_meta_bytes(cfg.stages) + size_t(cfg.stages) * cfg.stage_bytes + table +
                       (mode == kBmShared ? bitmap : mode == kBmCluster ? half : 0);
    switch (mode) {
    case kBmShared:
        return launch_q3_kern<W, kBmShared>(shm, cfg, kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, gt,
                                            hits, d_err, st);
    case kBmCluster:
        return launch_q3_kern<W, kBmCluster>(shm, cfg, kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, gt,
                                             hits, d_err, st);
    default:
        return launch_q3_kern<W, kBmGlobal>(shm, cfg, kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, gt,
                                            hits, d_err, st);
    }
}

int launch_q3_tma(const ColView &kv, const ColView &gv, const ColView &mv, const StreamCol &s0, const StreamCol &s1,
                  const StreamCol &s2, const StreamCol &s3, const Pred &pred, const uint32_t *bits, uint64_t nwords,
                  uint64_t lo, uint64_t span, const GTable &gt, uint32_t *hits, unsigned *d_err, cudaStream_t st) {
    switch (g_q3.warps) {
    case 8: return launch_q3_tma_w<8>(kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, gt, hits, d_err, st);
    case 24: return launch_q3_tma_w<24>(kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, gt, hits, d_err, st);
    default: return launch_q3_tma_w<16>(kv, gv, mv, s0, s1, s2, s3, pred, bits, nwords, lo, span, gt, hits, d_err, st);
    }
}

}  // namespace
}  // namespace ms

using namespace ms;

// Launch configuration of the fused query's staged kernel: staged (0 = the
// direct kernel only, 1 = staged with the build-side bitmap in shared memory
// when it fits beside the ring, 2 = staged with the bitmap in global memory,
// 3 = staged with the bitmap split over a 2-CTA cluster), warps
// (consumer warps: 8, 16 or 24), stages and
// stage_bytes (shared-memory ring; stages x stage_bytes + 48 KiB group table
// must fit 227 KiB).  The other fields are ignored.
extern "C" int ms_gpu_set_query_tuning(const ms_tuning *t) {
    if (!t) return ms_fail(MS_ERR_INVALID, "set_query_tuning: null");
    if (t->staged > 3) return ms_fail(MS_ERR_INVALID, "set_query_tuning: staged must be 0, 1, 2 or 3");
    if (t->warps != 8 && t->warps != 16 && t->warps != 24)
        return ms_fail(MS_ERR_INVALID, "set_query_tuning: warps must be 8, 16 or 24");
    if (t->stages < 2 || t->stages > 16 || t->stage_bytes % 128 || t->stage_bytes < 16384)
        return ms_fail(MS_ERR_INVALID, "set_query_tuning: stages in 2..16, stage_bytes a multiple of 128, >= 16 KiB");
    if (q3_meta_bytes(t->stages) + uint64_t(t->stages) * t->stage_bytes + 3ull * 8 * kQSlots > 232448)
        return ms_fail(MS_ERR_INVALID, "set_query_tuning: shared memory above 227 KiB");
    g_q3 = *t;
    return MS_OK;
}

extern "C" int ms_gpu_query3_last_pass_ms(double *ms) {
    if (!ms) return ms_fail(MS_ERR_INVALID, "query3_last_pass_ms: null");
    *ms = g_q3_pass_ms;
    return MS_OK;
}

extern "C" int ms_gpu_get_query_tuning(ms_tuning *t) {
    if (!t) return ms_fail(MS_ERR_INVALID, "get_query_tuning: null");
    *t = g_q3;
    return MS_OK;
}

// The fused query.  Outputs (host arrays of capacity `cap`): group keys, the
// group extents (first position of each group within P, as group_vec
// returns them) and the grouped sums, in group-id order; *n_groups.
// The build side `l` must span at most 2^30 values (a dense bitmap).
extern "C" int ms_gpu_query3(const ms_col *filter, int cmp, uint64_t c, const ms_col *fk, const ms_col *l,
                             const ms_col *gkey, const ms_col *measure, uint64_t cap, uint64_t *h_keys,
                             uint64_t *h_ext, uint64_t *h_sums, uint64_t *n_groups, uint64_t *n_rows_p,
                             ms_arena *a, void *stream) {
    if (!filter || !fk || !l || !gkey || !measure || !n_groups || !a) return ms_fail(MS_ERR_INVALID, "query3: null");
    const uint64_t n = filter->count_values;
    if (fk->count_values != n || gkey->count_values != n || measure->count_values != n)
        return ms_fail(MS_ERR_INVALID, "query3: fact columns differ in length");
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t mark0 = a->used;  // everything below is scratch
    ColView fv, kv, gv, mv, lv;
    int rc;
    if ((rc = prepare_view(filter, a, st, &fv)) || (rc = prepare_view(fk, a, st, &kv)) ||
        (rc = prepare_view(gkey, a, st, &gv)) || (rc = prepare_view(measure, a, st, &mv)) ||
        (rc = prepare_view(l, a, st, &lv)))
        return rc;
    // build side bitmap
    unsigned long long *mm = arena_take_t<unsigned long long>(a, 2);
    if (!mm) return ms_fail(MS_ERR_NOMEM, "arena exhausted (query3)");
    const unsigned grid = unsigned(maxu(1, minu((lv.nblocks_total() + 7) / 8, persistent_grid(256, 8))));
    uint64_t hmm[2] = {0, 0};
    if (lv.n && (rc = key_range(lv, mm, hmm, hmm + 1, a, st))) return rc;
    uint64_t lo = 0, span = 0;
    if (lv.n) {
        lo = hmm[0];
        if (hmm[1] - hmm[0] >= (uint64_t(1) << 30))
            return ms_fail(MS_ERR_UNSUPPORTED, "query3: build keys span more than 2^30");
        span = hmm[1] - hmm[0] + 1;
    }
    const uint64_t words = (span + 31) / 32 + 1;
    uint32_t *bits = arena_take_t<uint32_t>(a, words);
    if (!bits) return ms_fail(MS_ERR_NOMEM, "arena exhausted (query3)");
    MS_CUDA_TRY(cudaMemsetAsync(bits, 0, 4 * words, st));
    if (lv.n) {
        k_q3_bits<<<grid, 256, 0, st>>>(lv, lo, bits, a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
    }
    const uint64_t nbt = fv.nblocks_total();
    // The global group table starts at 2^16 slots and grows by 16x (up to
    // 2^24) when it fills, re-running the pass.
    uint64_t slots = uint64_t(1) << 16;
    std::vector<uint64_t> more;     // records beyond the first kQFirstGroups
    const uint64_t *rec = nullptr;  // (key, extent, sum, first row) per group
    uint64_t ng = 0, np = 0;
    for (;;) {
        const uint64_t mark = a->used;
        uint32_t *hits = arena_take_t<uint32_t>(a, nbt + 1);
        uint64_t *boff = arena_take_t<uint64_t>(a, nbt + 1);
        uint64_t *tot = arena_take_t<uint64_t>(a, 1);
        uint64_t *scr = arena_take_t<uint64_t>(a, scan_scratch_words(nbt));
        GTable gt{arena_take_t<unsigned long long>(a, slots), arena_take_t<unsigned long long>(a, slots),
                  arena_take_t<unsigned long long>(a, slots), slots - 1};
        unsigned long long *cnt = arena_take_t<unsigned long long>(a, 1);
        uint64_t *out = arena_take_t<uint64_t>(a, 4 * slots);
        if (!hits || !boff || !tot || !scr || !gt.keys || !gt.first || !gt.sums || !cnt || !out)
            return ms_fail(MS_ERR_NOMEM, "arena exhausted (query3)");
        MS_CUDA_TRY(cudaMemsetAsync(gt.keys, 0xFF, 8 * slots, st));
        MS_CUDA_TRY(cudaMemsetAsync(gt.first, 0xFF, 8 * slots, st));
        MS_CUDA_TRY(cudaMemsetAsync(gt.sums, 0, 8 * slots, st));
        MS_CUDA_TRY(cudaMemsetAsync(cnt, 0, 8, st));
        MS_CUDA_TRY(cudaMemsetAsync(tot, 0, 8, st));
        if (!g_q3_ev[0]) {
            MS_CUDA_TRY(cudaEventCreate(&g_q3_ev[0]));
            MS_CUDA_TRY(cudaEventCreate(&g_q3_ev[1]));
        }
        MS_CUDA_TRY(cudaEventRecord(g_q3_ev[0], st));
        if (nbt) {
            uint64_t nbs = 0;  // blocks through the staged kernel
            if (g_q3.staged && plain(fv) && random_access(kv) && random_access(gv) && random_access(mv)) {
                const StreamCol s0 = stream_of(fv), s1 = stream_of(kv), s2 = stream_of(gv), s3 = stream_of(mv);
                nbs = minu(minu(s0.nb, s1.nb), minu(s2.nb, s3.nb));
                if (nbs) {
                    rc = launch_q3_tma(kv, gv, mv, s0, s1, s2, s3, make_pred(cmp, c), bits, words, lo, span, gt,
                                       hits, a->d_err, st);
                    if (rc) return rc;
                }
            }
            if (nbt > nbs) {
                const unsigned g2 = unsigned(maxu(1, minu((nbt - nbs + 7) / 8, persistent_grid(256, 4))));
                k_query3<<<g2, 256, 0, st>>>(fv, kv, gv, mv, cmp, c, bits, lo, span, gt, hits, nbs, a->d_err);
                MS_CUDA_TRY(cudaGetLastError());
            }
            MS_CUDA_TRY(cudaEventRecord(g_q3_ev[1], st));
            MS_CUDA_TRY(scan_exclusive<uint32_t>(hits, nbt, boff, tot, scr, st));
            k_q3_extents<<<unsigned(minu(slots / 256, persistent_grid(256, 2))), 256, 0, st>>>(
                gt, fv, kv, cmp, c, bits, lo, span, boff, cnt, out, a->d_err);
            MS_CUDA_TRY(cudaGetLastError());
        }
        // counts, error word and the first kQFirstGroups records in one
        // read-back; more groups take a second copy
        const uint64_t first = minu(slots, kQFirstGroups);
        ReadBack back(a, st);
        const unsigned *herr = back.add(a->d_err);
        const unsigned long long *hng = back.add(cnt);
        const uint64_t *hnp = back.add(tot);
        if (nbt) rec = back.add(out, 4 * first);
        rc = back.wait_results();
        if (rc) return rc;
        if (*herr == kErrCapacity && slots < (uint64_t(1) << 24)) {
            MS_CUDA_TRY(cudaMemsetAsync(a->d_err, 0, sizeof *herr, st));
            a->used = mark;
            slots <<= 4;
            continue;
        }
        rc = error_status(*herr, a, st);
        if (rc) return rc;
        float pass_ms = 0;
        if (nbt && cudaEventElapsedTime(&pass_ms, g_q3_ev[0], g_q3_ev[1]) == cudaSuccess) g_q3_pass_ms = pass_ms;
        ng = *hng;
        np = *hnp;
        if (ng > first) {
            more.resize(4 * ng);
            std::copy(rec, rec + 4 * first, more.begin());
            MS_CUDA_TRY(cudaMemcpyAsync(more.data() + 4 * first, out + 4 * first, 32 * (ng - first),
                                        cudaMemcpyDeviceToHost, st));
            MS_CUDA_TRY(cudaStreamSynchronize(st));
            rec = more.data();
        }
        break;
    }
    a->used = mark0;
    // group ids follow the first occurrence: order by first row
    std::vector<uint64_t> idx(ng);
    for (uint64_t i = 0; i < ng; i++) idx[i] = i;
    std::sort(idx.begin(), idx.end(), [&](uint64_t x, uint64_t y) { return rec[4 * x + 3] < rec[4 * y + 3]; });
    *n_groups = ng;
    if (n_rows_p) *n_rows_p = np;
    if (ng > cap) return ms_fail(MS_ERR_NOMEM, "query3: more groups than the output capacity");
    for (uint64_t i = 0; i < ng; i++) {
        if (h_keys) h_keys[i] = rec[4 * idx[i]];
        if (h_ext) h_ext[i] = rec[4 * idx[i] + 1];
        if (h_sums) h_sums[i] = rec[4 * idx[i] + 2];
    }
    return MS_OK;
}
