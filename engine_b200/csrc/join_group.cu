// join_group.cu -- semi_join, intersect_sorted, group and grouped agg_sum
// with decompression fused into the probe / grouping kernels.
//
// Membership (semi_join build side): when the build keys span at most 2^27
// values the set is a dense bitmap (exact, one bit per value; kept in
// shared memory when it fits 208 KB), otherwise an open-addressing hash set
// in global memory (linear probing, 64-bit multiplicative hash).  The
// reference uses a vectorised linear-probing hash set
// (vector/datastructures/hash_based/hash_set.h:32-149); results do not
// depend on the table, only on set membership.
//
// Grouping: a global hash table maps each key to the smallest row where it
// occurs (atomicMin); flags at those rows, scanned, give every group its id
// in order of first occurrence -- exactly the reference's ids
// (linear_probing.h:437-443, scalar/group_uncompr.h:105-114) -- and the
// flagged rows in order are the group extents.
#include "internal.h"
#include "positions.cuh"
#include "scan.cuh"

namespace ms {

int gather_values(const ms_col *data, const uint64_t *d_pos, uint64_t npos, uint64_t *d_out, ms_arena *a,
                  cudaStream_t st);

namespace {

constexpr uint64_t kEmpty = ~uint64_t(0);

__device__ __forceinline__ uint64_t hash64(uint64_t k) {
    k ^= k >> 33;
    k *= 0xFF51AFD7ED558CCDull;
    k ^= k >> 33;
    k *= 0xC4CEB9FE1A85EC53ull;
    k ^= k >> 33;
    return k;
}

struct KeySet {
    // bitmap mode
    const uint32_t *bits;  // global bitmap (nullptr in hash mode)
    uint64_t lo;           // smallest key
    uint64_t span;         // bits in the bitmap
    // hash mode
    const uint64_t *slots;
    uint64_t mask;
    int has_max;           // key 2^64-1 present (it doubles as the empty marker)
};

__device__ __forceinline__ bool set_contains(const KeySet &s, const uint32_t *sbits, uint64_t k) {
    if (s.bits) {
        const uint64_t d = k - s.lo;
        if (k < s.lo || d >= s.span) return false;
        const uint32_t *b = sbits ? sbits : s.bits;
        return (b[d >> 5] >> (d & 31u)) & 1u;
    }
    if (k == kEmpty) return s.has_max;
    uint64_t h = hash64(k) & s.mask;
    for (uint64_t probe = 0; probe <= s.mask; probe++) {
        const uint64_t v = s.slots[h];
        if (v == k) return true;
        if (v == kEmpty) return false;
        h = (h + 1) & s.mask;
    }
    return false;
}

__global__ void k_build_set(ColView c, uint32_t *bits, uint64_t lo, uint64_t *slots, uint64_t mask,
                            int *has_max, unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < c.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16];
        unsigned valid;
        ok &= decode_block(c, b, l, q, v, valid);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            if (!((valid >> k) & 1u)) continue;
            const uint64_t key = v[k];
            if (bits) {
                const uint64_t d = key - lo;
                atomicOr(bits + (d >> 5), 1u << (d & 31u));
                continue;
            }
            if (key == kEmpty) {
                *has_max = 1;
                continue;
            }
            uint64_t h = hash64(key) & mask;
            bool placed = false;
            for (uint64_t probe = 0; probe <= mask; probe++) {
                const unsigned long long old =
                    atomicCAS((unsigned long long *)(slots + h), (unsigned long long)kEmpty, (unsigned long long)key);
                if (old == kEmpty || old == key) {
                    placed = true;
                    break;
                }
                h = (h + 1) & mask;
            }
            if (!placed) atomicOr(err, kErrCapacity);
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
}

// Probe, pass 1: hit bits = rows of r whose value is in the set.  A bitmap of
// up to kSmemBitmapWords is copied into shared memory by one CTA of 24 warps
// per SM (random words of global memory cost one L1 line each, 32 per warp
// load; shared memory serves them at its bank conflicts).  Blocks of width <=
// 32 are decoded to 32-bit values; a value's place in the bitmap is its
// distance from the smallest key, which is at or beyond the span for any
// value below that key.
constexpr unsigned kSmemBitmapWords = 53248;  // 208 KB
constexpr unsigned kProbeWarps = 24;

template <bool kSmem>
__global__ void __launch_bounds__(kSmem ? 32 * kProbeWarps : 256, kSmem ? 1 : 3)
    k_probe_bits(ColView r, KeySet s, MaskRun run, unsigned *err) {
    extern __shared__ uint32_t sbits[];
    if (kSmem) {
        const uint32_t words = uint32_t((s.span + 31) / 32);
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) sbits[i] = __ldg(s.bits + i);
        __syncthreads();
    }
    bool ok = true;
    const bool narrow = s.bits && (r.fmt == MS_FMT_STATIC_VBP || r.fmt == MS_FMT_DYNAMIC_VBP || r.fmt == MS_FMT_FOR_DVBP);
    mask_pass(run, [&](uint64_t b, unsigned l, unsigned q) -> unsigned {
        unsigned m = 0;
        if (narrow && b < r.nb()) {
            uint64_t off;
            unsigned bw;
            if (r.fmt == MS_FMT_STATIC_VBP) {
                bw = r.bw;
                off = b * 64ull * bw;
            } else {
                const uint64_t e = __ldg(r.index + b);
                off = idx_off(e);
                bw = idx_bw(e);
            }
            uint32_t v[16];
            if (vbp_decode16_u32_rt(bw, reinterpret_cast<const uint64_t *>(r.data + off), l, q, v)) {
                const uint64_t base = (r.fmt == MS_FMT_FOR_DVBP ? __ldg(r.aux + (b >> 1)) : 0) - s.lo;
#pragma unroll
                for (int k = 0; k < 16; k++) {
                    const uint64_t d = base + v[k];
                    const uint32_t w = d < s.span ? (kSmem ? sbits[uint32_t(d >> 5)] : __ldg(s.bits + (d >> 5))) : 0u;
                    m |= ((w >> (unsigned(d) & 31u)) & 1u) << k;
                }
                return m;
            }
        }
        uint64_t v[16];
        unsigned valid;
        ok &= decode_block(r, b, l, q, v, valid);
#pragma unroll
        for (int k = 0; k < 16; k++)
            if ((valid >> k) & 1u) m |= unsigned(set_contains(s, kSmem ? sbits : nullptr, v[k])) << k;
        return m;
    });
    if (!ok) atomicOr(err, kErrCorrupt);
}

// ---------------------------------------------------------------------------
// Natural equi-join (join_natural_equi_compr.h:116-300): the build side maps
// every key to the position of its first occurrence (the reference's hash
// map keeps the value of the first insert, linear_probing.h:315-366).  Dense
// key ranges use a direct array of positions, others an open-addressing
// table; both are filled with atomicMin, so the result does not depend on the
// order in which warps insert.
// ---------------------------------------------------------------------------
struct KeyMap {
    uint32_t *dense;      // dense mode: position per key - lo (~0: absent); builds of fewer than 2^32 - 1 rows
    uint32_t *bits;       // dense mode: keys present
    uint64_t lo, span;
    unsigned long long *keys;   // hash mode
    unsigned long long *vals;
    uint64_t mask;
    unsigned long long *max_pos;  // position of key 2^64-1 (it doubles as the empty marker)
};

__device__ __forceinline__ uint64_t map_lookup(const KeyMap &m, uint64_t k) {
    if (m.dense) {
        const uint64_t d = k - m.lo;
        if (d >= m.span) return kEmpty;
        const uint32_t p = m.dense[d];
        return p == ~0u ? kEmpty : p;
    }
    if (k == kEmpty) return *m.max_pos;
    uint64_t h = hash64(k) & m.mask;
    for (uint64_t probe = 0; probe <= m.mask; probe++) {
        const uint64_t v = m.keys[h];
        if (v == k) return m.vals[h];
        if (v == kEmpty) return kEmpty;
        h = (h + 1) & m.mask;
    }
    return kEmpty;
}

__global__ void k_build_map(ColView c, KeyMap m, unsigned *err) {
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < c.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16];
        unsigned valid;
        ok &= decode_block(c, b, l, q, v, valid);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            if (!((valid >> k) & 1u)) continue;
            const uint64_t key = v[k];
            const unsigned long long row = b * kBlock + (16u * q + k) * 8u + l;
            if (m.dense) {
                const uint64_t d = key - m.lo;
                atomicMin(m.dense + d, uint32_t(row));
                atomicOr(m.bits + (d >> 5), 1u << (d & 31u));
                continue;
            }
            if (key == kEmpty) {
                atomicMin(m.max_pos, row);
                continue;
            }
            uint64_t h = hash64(key) & m.mask;
            bool placed = false;
            for (uint64_t probe = 0; probe <= m.mask; probe++) {
                const unsigned long long old = atomicCAS(m.keys + h, (unsigned long long)kEmpty, (unsigned long long)key);
                if (old == kEmpty || old == key) {
                    atomicMin(m.vals + h, row);
                    placed = true;
                    break;
                }
                h = (h + 1) & m.mask;
            }
            if (!placed) atomicOr(err, kErrCapacity);
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
}

// Probe, pass 1: hit bits = rows of r whose value is a key, and the build
// positions of a block's hits one after another at side + 512 * block (V:
// 32 bits while positions fit).  kSmem: the bitmap of present keys in shared
// memory decides the rows, so that only hits read the position array (one
// L1 line per row otherwise, which is what bounds a probe of all rows).
template <bool kSmem, class V>
__global__ void __launch_bounds__(kSmem ? 32 * kProbeWarps : 256, kSmem ? 1 : 3)
    k_probe_map_bits(ColView r, KeyMap m, MaskRun run, V *__restrict__ side, unsigned *err) {
    extern __shared__ uint32_t sbits[];
    if (kSmem) {
        const uint32_t words = uint32_t((m.span + 31) / 32);
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) sbits[i] = __ldg(m.bits + i);
        __syncthreads();
    }
    bool ok = true;
    mask_pass(run, [&](uint64_t b, unsigned l, unsigned q) -> unsigned {
        uint64_t v[16];
        unsigned valid, mk = 0;
        ok &= decode_block(r, b, l, q, v, valid);
        V *const o = side + (b - run.b0) * kBlock;
        if (kSmem) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const uint64_t d = v[k] - m.lo;
                v[k] = d;
                if (d < m.span) mk |= ((sbits[uint32_t(d >> 5)] >> (unsigned(d) & 31u)) & 1u) << k;
            }
            mk &= valid;
        } else {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const uint64_t p = ((valid >> k) & 1u) ? map_lookup(m, v[k]) : kEmpty;
                v[k] = p;  // the build position replaces the value
                mk |= unsigned(p != kEmpty) << k;
            }
        }
        if (__any_sync(0xFFFFFFFFu, mk != 0)) {
            unsigned rank[16];
            block_ranks(mk, l, q, rank);
#pragma unroll
            for (int k = 0; k < 16; k++)
                if ((mk >> k) & 1u) o[rank[k]] = kSmem ? V(__ldg(m.dense + v[k])) : V(v[k]);
        }
        return mk;
    });
    if (!ok) atomicOr(err, kErrCorrupt);
}

// intersect, pass 1: hit bits = rows of l (a sorted position list) whose value
// occurs in the sorted array rv; the hits' values compact per block.  A warp
// finds the part of rv that its block's values span by two 32-way searches,
// copies it to shared memory when it has at most kIsectPart values, and runs
// the binary searches of a thread's 16 values side by side in it (in rv
// itself when the part is longer).  Two lists of 2^22.7 positions: 74 us, and
// 7 to collect the values; galloping searches in global memory, one value
// after another in two passes, took 401.
constexpr unsigned kIsectPart = 1024;

// first index in rv[lo, hi) with rv[i] >= x (kUpper: > x); all lanes together
template <bool kUpper>
__device__ __forceinline__ uint64_t warp_bound(const uint64_t *__restrict__ rv, uint64_t lo, uint64_t hi, uint64_t x,
                                               unsigned lane) {
    while (lo < hi) {
        const uint64_t step = (hi - lo + 31) / 32, p = lo + lane * step;
        const bool before = p < hi && (kUpper ? __ldg(rv + p) <= x : __ldg(rv + p) < x);
        const unsigned cnt = __popc(__ballot_sync(0xFFFFFFFFu, before));  // probes before the bound: a prefix
        if (cnt == 0) return lo;
        const uint64_t last = lo + (cnt - 1) * step;
        hi = minu(hi, last + step);
        lo = last + 1;
    }
    return lo;
}

// bit k: v[k] occurs in the sorted a[0, len), len > 0
template <class I>
__device__ __forceinline__ unsigned search16(const uint64_t *a, I len, const uint64_t (&v)[16]) {
    I at[16];
#pragma unroll
    for (int k = 0; k < 16; k++) at[k] = 0;
    for (I n = len; n > 1;) {
        const I h = n >> 1;
#pragma unroll
        for (int k = 0; k < 16; k++) at[k] += a[at[k] + h - 1] < v[k] ? h : 0;
        n -= h;
    }
    unsigned m = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) m |= unsigned(a[at[k]] == v[k]) << k;
    return m;
}

__global__ void __launch_bounds__(256, 3) k_intersect_bits(ColView lc, const uint64_t *__restrict__ rv, uint64_t nr,
                                                          MaskRun run, uint64_t *__restrict__ side, unsigned *err) {
    extern __shared__ __align__(16) uint64_t isect_smem[];
    uint64_t *const part = isect_smem + (threadIdx.x >> 5) * kIsectPart;
    bool ok = true;
    mask_pass(run, [&](uint64_t b, unsigned l, unsigned q) -> unsigned {
        const unsigned lane = threadIdx.x & 31u;
        uint64_t v[16];
        unsigned valid, m = 0;
        ok &= decode_block(lc, b, l, q, v, valid);
        // the block's last value: the largest of the valid ones
        uint64_t hi_v = 0;
#pragma unroll
        for (int k = 0; k < 16; k++)
            if ((valid >> k) & 1u) hi_v = maxu(hi_v, v[k]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) hi_v = maxu(hi_v, __shfl_xor_sync(0xFFFFFFFFu, hi_v, d));
        const uint64_t lo_v = __shfl_sync(0xFFFFFFFFu, v[0], 0);
        const uint64_t lo = warp_bound<false>(rv, 0, nr, lo_v, lane), hi = warp_bound<true>(rv, lo, nr, hi_v, lane);
        if (lo < hi) {
            const uint64_t len = hi - lo;
            if (len <= kIsectPart) {
                for (unsigned i = lane; i < len; i += 32) part[i] = __ldg(rv + lo + i);
                __syncwarp();
                m = search16<unsigned>(part, unsigned(len), v);
            } else {
                m = search16<uint64_t>(rv + lo, len, v);
            }
            m &= valid;
            __syncwarp();  // the part is free for the warp's next block
        }
        if (__any_sync(0xFFFFFFFFu, m != 0)) {
            uint64_t *const o = side + (b - run.b0) * kBlock;
            unsigned rank[16];
            block_ranks(m, l, q, rank);
#pragma unroll
            for (int k = 0; k < 16; k++)
                if ((m >> k) & 1u) o[rank[k]] = v[k];
        }
        return m;
    });
    if (!ok) atomicOr(err, kErrCorrupt);
}

// --- group ------------------------------------------------------------------
// Global group table (open addressing).  An entry is empty until `first` is
// set: the inserter that claims the slot (state 0 -> 1) writes the key, then
// publishes it by storing its row in `first`; later rows of the key only ever
// lower `first`.  After the insert pass `state` holds group id + 1 (0: empty).
struct GroupEntry {
    uint64_t ka;               // key (unary) / group (binary)
    unsigned long long first;  // smallest row of the key, ~0 until the key is written
};

struct GroupTable {
    GroupEntry *e;
    uint64_t *kb;              // value (binary) or nullptr
    unsigned *state;
    unsigned long long *fill;  // claimed slots
    uint64_t mask;
    uint64_t limit;            // claims allowed before the table counts as full
};

__device__ __forceinline__ uint64_t hash_pair(uint64_t a, uint64_t b) { return hash64(a * 0x9E3779B97F4A7C15ull ^ b); }

enum { kInsOk = 0, kInsFull = 1, kInsTimeout = 2 };

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Insert (key, row).  A published slot costs loads only: the key is compared
// and `first` lowered by atomicMin only when the row is smaller, which for
// rows taken in ascending order is rare -- an atomic per row serialised the
// frequent keys of a skewed column.
__device__ __forceinline__ int group_insert(const GroupTable &t, uint64_t a, uint64_t b, uint64_t row) {
    uint64_t h = hash_pair(a, b) & t.mask;
    for (uint64_t probe = 0; probe <= t.mask; probe++) {
        GroupEntry *const e = t.e + h;
        unsigned long long f = ld_acquire(&e->first);
        if (f == kEmpty) {
            if (atomicCAS(t.state + h, 0u, 1u) == 0u) {
                if (atomicAdd(t.fill, 1ull) >= t.limit) {
                    atomicExch(t.state + h, 0u);
                    return kInsFull;
                }
                e->ka = a;
                if (t.kb) t.kb[h] = b;
                __threadfence();
                atomicMin(&e->first, (unsigned long long)row);
                return kInsOk;
            }
            // another inserter is writing the key (or gave the slot back: the
            // table is full)
            for (unsigned spins = 0; f == kEmpty; spins++) {
                if (spins >= kSpinLimit) return kInsTimeout;
                if (*(volatile unsigned long long *)t.fill > t.limit) return kInsFull;
                f = ld_acquire(&e->first);
            }
        }
        if (((volatile uint64_t *)&e->ka)[0] == a && (!t.kb || ((volatile uint64_t *)t.kb)[h] == b)) {
            if (row < f) atomicMin(&e->first, (unsigned long long)row);
            return kInsOk;
        }
        h = (h + 1) & t.mask;
    }
    return kInsFull;
}

// pass A: every row's key with its row number.  Each CTA first folds its rows
// into a shared-memory table (key -> smallest row seen by the CTA; a few
// shared loads per row, no atomics once a key is in), and inserts that table
// into the global one at the end.  Keys that find no place among kGrpProbes
// slots go to the global table row by row, and a warp whose block mostly
// missed stops asking the shared table (many distinct keys).  Bound by the
// shared-memory lookups.  2^25 rows, 1000 Zipf(1.1) keys: 0.149 ms; with a
// global compare-and-swap and minimum per row 11.1 ms, and 6.3 ms before it
// for a first attempt in a table too small for the keys.
constexpr unsigned kGrpSlots = 4096, kGrpProbes = 8;

__device__ __forceinline__ unsigned grp_hash(uint64_t a) {
    const uint32_t x = uint32_t(a) ^ (uint32_t(a >> 32) * 0x85EBCA6Bu);
    return ((x ^ (x >> 15)) * 0x9E3779B1u) >> 20;  // 12 bits
}

// slot h of a shared table as one 16-byte load
__device__ __forceinline__ ulonglong2 slot_ld(const unsigned long long *table, unsigned h) {
    ulonglong2 v;
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                 : "=l"(v.x), "=l"(v.y)
                 : "r"(uint32_t(__cvta_generic_to_shared(table + 2 * h))));
    return v;
}

template <bool kBinary>
__global__ void __launch_bounds__(256, 3) k_group_insert(ColView gin, ColView c, GroupTable t, unsigned *err) {
    extern __shared__ __align__(16) unsigned long long grp_smem[];  // unary: (key, smallest row) slots, ~0 empty
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    if (!kBinary) {
        for (unsigned i = threadIdx.x; i < 2 * kGrpSlots; i += blockDim.x) grp_smem[i] = kEmpty;
        __syncthreads();
    }
    bool ok = true, bypass = kBinary;
    int bad = kInsOk;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < c.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16], g[16];
        unsigned valid, vg, missed = 0;
        ok &= decode_block(c, b, l, q, v, valid);
        if (kBinary) ok &= decode_block(gin, b, l, q, g, vg);
        const uint64_t row0 = b * kBlock + 128u * q + l;
        unsigned todo = valid;  // rows that the shared table has not settled
        if (!bypass) {
            // four first probes in flight; a row is settled when its key is
            // there with a row at or before it
#pragma unroll
            for (int k0 = 0; k0 < 16; k0 += 4) {
                ulonglong2 x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = slot_ld(grp_smem, grp_hash(v[k0 + i]));
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (x[i].x == v[k0 + i] && x[i].y <= row0 + 8u * (k0 + i)) todo &= ~(1u << (k0 + i));
            }
        }
        if (__any_sync(0xFFFFFFFFu, todo != 0)) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                if (!((todo >> k) & 1u)) continue;
                const uint64_t row = row0 + 8u * k;
                bool done = false;
                if (!bypass && v[k] != kEmpty) {
                    unsigned h = grp_hash(v[k]);
                    for (unsigned p = 0; p < kGrpProbes && !done; p++) {
                        unsigned long long *const e = grp_smem + 2 * h;
                        unsigned long long x = *(volatile unsigned long long *)e;
                        if (x == kEmpty) x = atomicCAS(e, (unsigned long long)kEmpty, (unsigned long long)v[k]);
                        if (x == kEmpty || x == v[k]) {
                            if (row < *(volatile unsigned long long *)(e + 1)) atomicMin(e + 1, (unsigned long long)row);
                            done = true;
                        }
                        h = (h + 1) & (kGrpSlots - 1);
                    }
                }
                if (!done) {
                    missed++;
                    if (bad == kInsOk) bad = kBinary ? group_insert(t, g[k], v[k], row) : group_insert(t, v[k], 0, row);
                }
            }
        }
        if (!kBinary) bypass |= __reduce_add_sync(0xFFFFFFFFu, missed) > kBlock / 2;
        if (__any_sync(0xFFFFFFFFu, bad != kInsOk)) break;
    }
    if (!kBinary) {
        __syncthreads();
        for (unsigned i = threadIdx.x; i < kGrpSlots && bad == kInsOk; i += blockDim.x)
            if (grp_smem[2 * i] != kEmpty) bad = group_insert(t, grp_smem[2 * i], 0, grp_smem[2 * i + 1]);
    }
    if (!ok) atomicOr(err, kErrCorrupt);
    if (bad == kInsFull) atomicOr(err, kErrCapacity);
    if (bad == kInsTimeout) atomicOr(err, kErrTimeout);
}

// --- pass B: group ids = ranks of the groups' first rows, extents = the first
// rows in order.  cnt[0] collects the number of list entries, cnt[1] the
// groups opened at rows >= sfrom (the scalar remainder).
// Few groups: their (first row, slot) pairs are listed and ranked by counting
// smaller first rows.
constexpr unsigned kRankGroups = 4096;

__global__ void k_group_list(GroupTable t, uint64_t sfrom, unsigned long long *__restrict__ cnt,
                             ulonglong2 *__restrict__ list) {
    for (uint64_t h = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; h <= t.mask; h += uint64_t(gridDim.x) * blockDim.x) {
        const unsigned long long r = t.e[h].first;
        if (r == kEmpty) continue;
        if (r >= sfrom) atomicAdd(cnt + 1, 1ull);
        if (list) list[atomicAdd(cnt, 1ull)] = make_ulonglong2(r, h);
    }
}

__global__ void __launch_bounds__(256) k_group_rank(GroupTable t, const ulonglong2 *__restrict__ list, unsigned ng,
                                                    uint64_t *__restrict__ ext) {
    __shared__ unsigned long long s_first[kRankGroups];
    for (unsigned i = threadIdx.x; i < ng; i += blockDim.x) s_first[i] = list[i].x;
    __syncthreads();
    // eight threads per group, 32 groups per CTA
    const unsigned i = blockIdx.x * 32u + threadIdx.x / 8u;
    const unsigned long long f = i < ng ? s_first[i] : 0;
    unsigned rank = 0;
    for (unsigned j = threadIdx.x & 7u; j < ng; j += 8u) rank += s_first[j] < f;
    rank += __shfl_xor_sync(0xFFFFFFFFu, rank, 1);
    rank += __shfl_xor_sync(0xFFFFFFFFu, rank, 2);
    rank += __shfl_xor_sync(0xFFFFFFFFu, rank, 4);
    if (i < ng && (threadIdx.x & 7u) == 0) {
        ext[rank] = f;
        t.state[list[i].y] = rank + 1;
    }
}

// Many groups: flags at the first rows (bitmap over rows), scanned.
__global__ void k_group_flags(GroupTable t, uint32_t *__restrict__ flags) {
    for (uint64_t h = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; h <= t.mask; h += uint64_t(gridDim.x) * blockDim.x) {
        const unsigned long long r = t.e[h].first;
        if (r != kEmpty) atomicOr(flags + (r >> 5), 1u << (r & 31u));
    }
}

__global__ void k_popc_words(const uint32_t *__restrict__ flags, uint64_t nwords, uint32_t *__restrict__ cnt) {
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nwords; i += uint64_t(gridDim.x) * blockDim.x)
        cnt[i] = __popc(flags[i]);
}

// extents: the first rows in order; ids into the table
__global__ void k_group_extents(GroupTable t, const uint32_t *__restrict__ flags, const uint64_t *__restrict__ woff,
                                uint64_t *__restrict__ ext) {
    for (uint64_t h = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; h <= t.mask; h += uint64_t(gridDim.x) * blockDim.x) {
        const unsigned long long r = t.e[h].first;
        if (r == kEmpty) continue;
        const uint64_t id = woff[r >> 5] + __popc(flags[r >> 5] & ((1u << (r & 31u)) - 1u));
        ext[id] = r;
        t.state[h] = unsigned(id) + 1u;
    }
}

// pass C: group id of every row.  Unary columns of up to kGrpSmemGroups
// groups are looked up in a shared-memory copy of the table (key -> id);
// others, and keys that found no place there, in the global table.
// 2^25 rows, 1000 keys: 0.111 ms (0.325 ms with every row looked up in the
// global table and its flags; writing the ids alone takes 0.041 ms).
constexpr unsigned kGrpSmemGroups = kGrpSlots / 2;

__device__ __forceinline__ unsigned group_find(const GroupTable &t, uint64_t a, uint64_t b) {
    uint64_t h = hash_pair(a, b) & t.mask;
    for (uint64_t probe = 0; probe <= t.mask; probe++) {
        const unsigned id = __ldg(t.state + h);
        if (id == 0) return 0;
        if (__ldg(&t.e[h].ka) == a && (!t.kb || __ldg(t.kb + h) == b)) return id;
        h = (h + 1) & t.mask;
    }
    return 0;
}

template <bool kBinary>
__global__ void __launch_bounds__(256, 3) k_group_ids(ColView gin, ColView c, GroupTable t,
                                                     const ulonglong2 *__restrict__ list, unsigned ng,
                                                     uint64_t *__restrict__ gr, unsigned *err) {
    extern __shared__ __align__(16) unsigned long long grp_smem[];
    // (key, id) slots, ~0 empty
    const bool smem = !kBinary && list != nullptr;
    if (smem) {
        for (unsigned i = threadIdx.x; i < 2 * kGrpSlots; i += blockDim.x) grp_smem[i] = kEmpty;
        __syncthreads();
        for (unsigned i = threadIdx.x; i < ng; i += blockDim.x) {
            const uint64_t slot = list[i].y, key = t.e[slot].ka;
            if (key == kEmpty) continue;
            unsigned h = grp_hash(key);
            for (unsigned p = 0; p < kGrpProbes; p++) {
                if (atomicCAS(grp_smem + 2 * h, (unsigned long long)kEmpty, (unsigned long long)key) == kEmpty) {
                    grp_smem[2 * h + 1] = t.state[slot];
                    break;
                }
                h = (h + 1) & (kGrpSlots - 1);
            }
        }
        __syncthreads();
    }
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < c.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t v[16], g[16];
        unsigned valid, vg;
        ok &= decode_block(c, b, l, q, v, valid);
        if (kBinary) ok &= decode_block(gin, b, l, q, g, vg);
        uint64_t *const out = gr + b * kBlock + 128u * q + l;
#pragma unroll
        for (int k0 = 0; k0 < 16; k0 += 4) {
            ulonglong2 x[4];
            if (smem) {
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = slot_ld(grp_smem, grp_hash(v[k0 + i]));
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int k = k0 + i;
                if (!((valid >> k) & 1u)) continue;
                unsigned id = 0;
                if (smem && v[k] != kEmpty) {
                    unsigned h = grp_hash(v[k]);
                    for (unsigned p = 0;; p++) {
                        if (x[i].x == v[k]) id = unsigned(x[i].y);
                        if (x[i].x == v[k] || x[i].x == kEmpty || p + 1 == kGrpProbes) break;
                        h = (h + 1) & (kGrpSlots - 1);
                        x[i] = slot_ld(grp_smem, h);
                    }
                }
                if (id == 0) id = kBinary ? group_find(t, g[k], v[k]) : group_find(t, v[k], 0);
                ok &= id != 0;
                out[8u * k] = uint64_t(id) - 1u;
            }
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
}

// --- grouped sum ----------------------------------------------------------------
// Up to kSumSmemGroups groups: 64-bit sums as two 32-bit words per group in
// shared memory (32-bit shared atomics are native, 64-bit ones a CAS loop); a
// row adds its low word, and its high word plus the carry when that is not
// zero.  Few groups get several copies, one per lane & (copies - 1), so that
// the lanes of a warp that hit one frequent group do not serialise; an odd
// copy stride puts a group's copies in different banks.  2^25 rows, 1000
// Zipf(1.1) groups: 0.103 ms (0.726 ms with the lanes of equal groups combined
// by shuffles first).
constexpr unsigned kSumCopyBytes = 32768;    // copies are made while they fit this
constexpr unsigned kSumSmemGroups = 24576;   // 192 KB of sums
constexpr unsigned kSumSlots = 4096;         // (group + 1, low, high) slots of a CTA beyond that

__device__ __forceinline__ void sum_add(unsigned *s_lo, unsigned *s_hi, unsigned i, uint64_t d) {
    const unsigned lo = unsigned(d);
    const unsigned old = lo ? atomicAdd(s_lo + i, lo) : 0u;
    const unsigned hi = unsigned(d >> 32) + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd(s_hi + i, hi);
}

__global__ void __launch_bounds__(768, 1) k_grouped_sum(ColView gc, ColView dc, uint64_t ngroups, unsigned copies,
                                                       unsigned stride, unsigned long long *__restrict__ out,
                                                       unsigned *err) {
    extern __shared__ __align__(16) unsigned sum_smem[];
    unsigned *const s_lo = sum_smem, *const s_hi = sum_smem + copies * stride;
    for (unsigned i = threadIdx.x; i < 2 * copies * stride; i += blockDim.x) sum_smem[i] = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    const unsigned mine = (lane & (copies - 1)) * stride;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < gc.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t g[16], d[16];
        unsigned vg, vd;
        ok &= decode_block(gc, b, l, q, g, vg);
        ok &= decode_block(dc, b, l, q, d, vd);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            if (!((vg >> k) & 1u)) continue;
            if (g[k] >= ngroups) {
                ok = false;
                continue;
            }
            sum_add(s_lo, s_hi, mine + unsigned(g[k]), d[k]);
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
    __syncthreads();
    for (unsigned i = threadIdx.x; i < ngroups; i += blockDim.x) {
        unsigned long long s = 0;
        for (unsigned c = 0; c < copies; c++)
            s += ((unsigned long long)s_hi[c * stride + i] << 32) + s_lo[c * stride + i];
        if (s) atomicAdd(out + i, s);
    }
}

// More groups than that: a CTA sums the groups that find one of two slots of
// its own, first come, first served -- a group of more than a few in 10^4 rows
// is seen while slots are free -- and adds the other rows to the global
// sums.  Rows of one group that meet in a warp there (a group that became
// frequent when the slots were taken) are added up by shuffles first: the
// global sums take about one add per cycle and address.  2^23 rows, 30000
// groups, one of them in 90 % of the rows: 86 us a call, even groups 101,
// Zipf(1.1) 99 (with one global add per row 4840, 101 and 1910; with the equal
// lanes of every warp combined first 274, 227 and 1130).
__global__ void __launch_bounds__(256, 3) k_grouped_sum_many(ColView gc, ColView dc, uint64_t ngroups,
                                                            unsigned long long *__restrict__ out, unsigned *err) {
    extern __shared__ __align__(16) unsigned sum_smem[];
    unsigned *const s_tag = sum_smem, *const s_lo = sum_smem + kSumSlots, *const s_hi = sum_smem + 2 * kSumSlots;
    for (unsigned i = threadIdx.x; i < 3 * kSumSlots; i += blockDim.x) sum_smem[i] = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u, l = lane & 7u, q = lane >> 3;
    bool ok = true;
    for (uint64_t b = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; b < gc.nblocks_total();
         b += uint64_t(gridDim.x) * blockDim.x / 32) {
        uint64_t g[16], d[16];
        unsigned vg, vd;
        ok &= decode_block(gc, b, l, q, g, vg);
        ok &= decode_block(dc, b, l, q, d, vd);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            bool left = (vg >> k) & 1u;  // not added yet
            if (left && g[k] >= ngroups) {
                ok = false;
                left = false;
            }
            if (left && g[k] < 0xFFFFFFFFull) {
                const unsigned tag = unsigned(g[k]) + 1u;
                unsigned h = (unsigned(g[k]) * 0x9E3779B1u) >> 20;  // 12 bits
#pragma unroll
                for (int p = 0; p < 2 && left; p++, h ^= 1u) {
                    unsigned x = *(volatile unsigned *)(s_tag + h);
                    if (x == 0) x = atomicCAS(s_tag + h, 0u, tag);
                    if (x == 0 || x == tag) {
                        sum_add(s_lo, s_hi, h, d[k]);
                        left = false;
                    }
                }
            }
            const unsigned rest = __ballot_sync(0xFFFFFFFFu, left);
            if (!rest) continue;
            const int lead = __ffs(rest) - 1;
            const uint64_t lead_g = __shfl_sync(0xFFFFFFFFu, g[k], lead);  // all lanes take part
            const bool with = left && g[k] == lead_g;
            if (__popc(__ballot_sync(0xFFFFFFFFu, with)) >= 4) {
                uint64_t s = with ? d[k] : 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
                if (int(lane) == lead) atomicAdd(out + g[k], (unsigned long long)s);
                left = left && !with;
            }
            if (left) atomicAdd(out + g[k], (unsigned long long)d[k]);
        }
    }
    if (!ok) atomicOr(err, kErrCorrupt);
    __syncthreads();
    for (unsigned i = threadIdx.x; i < kSumSlots; i += blockDim.x)
        if (s_tag[i]) atomicAdd(out + (s_tag[i] - 1u), ((unsigned long long)s_hi[i] << 32) + s_lo[i]);
}

}  // namespace

static unsigned grid_blocks(uint64_t nbt) {
    return (unsigned)maxu(1, minu((nbt + 7) / 8, persistent_grid(256, 8)));
}

// Dynamic shared memory that a kernel may be launched with.  The limit belongs to
// the function, not to a launch, so it is always the kernel's largest: one
// thread's smaller size would fail another thread's launch.
template <class... P> static int allow_smem(void (*kern)(P...), unsigned most) {
    MS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most)));
    return MS_OK;
}

// The bitmap goes to shared memory when it fits and the probe side is long
// enough to pay for each SM's copy: an SM copies `words` and then looks up
// its share of the rows, one word each.
static bool smem_bitmap(uint64_t words, uint64_t nbt) {
    return words <= kSmemBitmapWords && words * uint64_t(sm_count()) <= nbt * kBlock;
}

static int view_or_decompress(const ms_col *c, ms_arena *a, cudaStream_t st, ColView *v) {
    if (c->format != MS_FMT_RLE) return prepare_view(c, a, st, v);
    uint64_t *tmp = arena_take_t<uint64_t>(a, c->count_values + 1);
    if (!tmp) return ms_fail(MS_ERR_NOMEM, "arena exhausted (rle)");
    int rc = decompress_to(c, tmp, a, st);
    if (rc) return rc;
    *v = ColView{};
    v->fmt = MS_FMT_UNCOMPR;
    v->n = c->count_values;
    v->rest = tmp;
    v->sfrom = v->n - v->n % kStep;
    return MS_OK;
}

}  // namespace ms

using namespace ms;

extern "C" int ms_gpu_semi_join(const ms_col *l, const ms_col *r, int out_format, unsigned out_bw, ms_col *out,
                                ms_arena *a, void *stream) {
    if (!l || !r || !out || !a) return ms_fail(MS_ERR_INVALID, "semi_join: null argument");
    if (r->format == MS_FMT_RLE) return ms_fail(MS_ERR_UNSUPPORTED, "semi_join: rle_f probe side");
    cudaStream_t st = (cudaStream_t)stream;
    ColView lv, rv;
    int rc = view_or_decompress(l, a, st, &lv);
    if (rc) return rc;
    rc = prepare_view(r, a, st, &rv);
    if (rc) return rc;
    // build side range
    unsigned long long *mm = arena_take_t<unsigned long long>(a, 2);
    int *has_max = arena_take_t<int>(a, 1);
    if (!mm || !has_max) return ms_fail(MS_ERR_NOMEM, "arena exhausted (semi_join)");
    const uint64_t nbl = lv.nblocks_total();
    uint64_t hmm[2] = {0, 0};
    if (nbl) {
        rc = key_range(lv, mm, hmm, hmm + 1, a, st);
        if (rc) return rc;
    }
    KeySet s{};
    const uint64_t nl = l->count_values;
    const bool bitmap = nl > 0 && (hmm[1] - hmm[0]) < (uint64_t(1) << 27);
    if (nl == 0) {
        s.bits = nullptr;
        s.slots = nullptr;
        s.mask = 0;
        uint64_t *one = arena_take_t<uint64_t>(a, 1);
        if (!one) return ms_fail(MS_ERR_NOMEM, "arena exhausted (semi_join)");
        MS_CUDA_TRY(cudaMemsetAsync(one, 0xFF, 8, st));
        s.slots = one;
    } else if (bitmap) {
        s.lo = hmm[0];
        s.span = hmm[1] - hmm[0] + 1;
        const uint64_t words = (s.span + 31) / 32;
        uint32_t *bits = arena_take_t<uint32_t>(a, words);
        if (!bits) return ms_fail(MS_ERR_NOMEM, "arena exhausted (semi_join bitmap)");
        MS_CUDA_TRY(cudaMemsetAsync(bits, 0, 4 * words, st));
        s.bits = bits;
        k_build_set<<<grid_blocks(nbl), 256, 0, st>>>(lv, bits, s.lo, nullptr, 0, has_max, a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
    } else {
        uint64_t cap = 16;
        while (cap < 2 * nl) cap <<= 1;
        uint64_t *slots = arena_take_t<uint64_t>(a, cap);
        if (!slots) return ms_fail(MS_ERR_NOMEM, "arena exhausted (semi_join table)");
        MS_CUDA_TRY(cudaMemsetAsync(slots, 0xFF, 8 * cap, st));
        s.slots = slots;
        s.mask = cap - 1;
        MS_CUDA_TRY(cudaMemsetAsync(has_max, 0, 4, st));
        k_build_set<<<grid_blocks(nbl), 256, 0, st>>>(lv, nullptr, 0, slots, s.mask, has_max, a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
        ReadBack back(a, st);
        const int *hm = back.add(has_max);
        rc = back.wait_results();
        if (rc) return rc;
        s.has_max = *hm;
    }
    const uint64_t words = (s.span + 31) / 32;
    const uint64_t nbt = rv.nblocks_total();
    const bool smem = s.bits && smem_bitmap(words, nbt);
    if (smem) {
        rc = allow_smem(k_probe_bits<true>, 4 * kSmemBitmapWords);
        if (rc) return rc;
    }
    auto pass1 = [&](const MaskRun &run, uint32_t *) {
        if (smem)
            k_probe_bits<true><<<mask_grid(run.nblk, kProbeWarps, 1), 32 * kProbeWarps, 4 * words, st>>>(rv, s, run,
                                                                                                    a->d_err);
        else
            k_probe_bits<false><<<mask_grid(run.nblk, 8, 3), 256, 0, st>>>(rv, s, run, a->d_err);
    };
    uint64_t *pos, cnt, nscal;
    rc = rows_by_mask<kRows, uint32_t>(rv, pass1, &pos, nullptr, &cnt, &nscal, a, st);
    if (rc) return rc;
    return write_values(pos, cnt - nscal, nscal, out_format, out_bw, out, a, st);
}

extern "C" int ms_gpu_intersect_sorted(const ms_col *l, const ms_col *r, int out_format, unsigned out_bw, ms_col *out,
                                       ms_arena *a, void *stream) {
    if (!l || !r || !out || !a) return ms_fail(MS_ERR_INVALID, "intersect_sorted: null argument");
    if (l->format == MS_FMT_RLE) return ms_fail(MS_ERR_UNSUPPORTED, "intersect_sorted: rle_f input");
    cudaStream_t st = (cudaStream_t)stream;
    ColView lv;
    int rc = prepare_view(l, a, st, &lv);
    if (rc) return rc;
    const uint64_t *rvals = (const uint64_t *)r->data;
    if (r->format != MS_FMT_UNCOMPR) {
        uint64_t *tmp = arena_take_t<uint64_t>(a, r->count_values + 1);
        if (!tmp) return ms_fail(MS_ERR_NOMEM, "arena exhausted (intersect)");
        rc = decompress_to(r, tmp, a, st);
        if (rc) return rc;
        rvals = tmp;
    } else {
        rc = check_col(r, false);
        if (rc) return rc;
    }
    const uint64_t nr = r->count_values;
    constexpr size_t smem = 8 * size_t(kIsectPart) * 8;
    MS_CUDA_TRY(cudaFuncSetAttribute(k_intersect_bits, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    auto pass1 = [&](const MaskRun &run, uint64_t *side) {
        k_intersect_bits<<<mask_grid(run.nblk, 8, 3), 256, smem, st>>>(lv, rvals, nr, run, side, a->d_err);
    };
    uint64_t *vals, cnt, nscal;
    rc = rows_by_mask<kVals, uint64_t>(lv, pass1, nullptr, &vals, &cnt, &nscal, a, st);
    if (rc) return rc;
    return write_values(vals, cnt - nscal, nscal, out_format, out_bw, out, a, st);
}

extern "C" int ms_gpu_group(const ms_col *gr_in, const ms_col *in, int gr_format, ms_col *out_gr, int ext_format,
                            ms_col *out_ext, ms_arena *a, void *stream) {
    if (!in || !out_gr || !out_ext || !a) return ms_fail(MS_ERR_INVALID, "group: null argument");
    if (gr_in && gr_in->count_values != in->count_values)
        return ms_fail(MS_ERR_INVALID, "binary group: inGrCol and inDataCol must contain the same number of data elements");
    cudaStream_t st = (cudaStream_t)stream;
    ColView cv, gv{};
    int rc = view_or_decompress(in, a, st, &cv);
    if (rc) return rc;
    if (gr_in) {
        rc = view_or_decompress(gr_in, a, st, &gv);
        if (rc) return rc;
    }
    const uint64_t n = in->count_values;
    const uint64_t nbt = cv.nblocks_total();
    // rows of the input's scalar remainder, and the groups they open, are
    // appended uncompressed (group_compr.h:136-265)
    const uint64_t sf = gr_in ? minu(cv.sfrom, gv.sfrom) : cv.sfrom;
    const bool binary = gr_in != nullptr;
    // 2^16 slots hold 2^15 groups; fewer when the column cannot have as many
    // groups or the arena is short.  A size that was found too small (below
    // `least`) is not tried again, so the table is filled once per size at
    // most.
    uint64_t cap = 1024, least = cap;
    while (cap < (uint64_t(1) << 16) && cap < 2 * n) cap <<= 1;
    const uint64_t mark = a->used;
    for (;;) {
        a->used = mark;
        GroupTable t{};
        t.e = arena_take_t<GroupEntry>(a, cap);
        t.kb = binary ? arena_take_t<uint64_t>(a, cap) : nullptr;
        t.state = arena_take_t<unsigned>(a, cap);
        unsigned long long *words = arena_take_t<unsigned long long>(a, 3);  // fill, list length, remainder groups
        t.fill = words;
        t.mask = cap - 1;
        t.limit = cap / 2;
        if (!t.e || !t.state || !words || (binary && !t.kb)) {
            if (cap > least) {
                cap >>= 1;
                continue;
            }
            return ms_fail(MS_ERR_NOMEM, "arena exhausted (group table)");
        }
        MS_CUDA_TRY(cudaMemsetAsync(t.e, 0xFF, sizeof(GroupEntry) * cap, st));
        MS_CUDA_TRY(cudaMemsetAsync(t.state, 0, 4 * cap, st));
        MS_CUDA_TRY(cudaMemsetAsync(words, 0, 24, st));
        constexpr size_t smem = 16 * kGrpSlots;
        if (nbt) {
            const unsigned grid = unsigned(minu((nbt + 7) / 8, persistent_grid(256, 3)));
            if (binary) {
                k_group_insert<true><<<grid, 256, 0, st>>>(gv, cv, t, a->d_err);
            } else {
                MS_CUDA_TRY(cudaFuncSetAttribute(k_group_insert<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 int(smem)));
                k_group_insert<false><<<grid, 256, smem, st>>>(gv, cv, t, a->d_err);
            }
            MS_CUDA_TRY(cudaGetLastError());
        }
        ReadBack back(a, st);
        const unsigned long long *h_groups = back.add(t.fill);
        rc = back.wait();
        if (rc == MS_ERR_NOMEM && cap < 4 * n + 4096) {
            least = 2 * cap;  // more distinct keys than the table holds: grow and redo
            cap *= 8;
            continue;
        }
        if (rc) return rc;
        const uint64_t groups = *h_groups;
        // the smallest table of that many groups, when it is smaller
        const auto shrink = [&] {
            while (least < 2 * groups) least <<= 1;
            if (cap == least) return false;
            cap = least;
            return true;
        };
        // The outputs, and for the ranking a list of few groups or flags per
        // row.  If neither fits beside the outputs, or their compressed form
        // does not, the call is made again with a smaller table.
        uint64_t *ext = arena_take_t<uint64_t>(a, groups + 1), *gr = arena_take_t<uint64_t>(a, n + 1);
        const uint64_t nwords = (n + 31) / 32;
        ulonglong2 *list = groups && groups <= kRankGroups ? arena_take_t<ulonglong2>(a, groups) : nullptr;
        uint32_t *flags = nullptr, *wcnt = nullptr;
        uint64_t *woff = nullptr, *tot = nullptr, *scr = nullptr;
        if (groups && !list) {
            flags = arena_take_t<uint32_t>(a, nwords + 1);
            wcnt = arena_take_t<uint32_t>(a, nwords + 1);
            woff = arena_take_t<uint64_t>(a, nwords + 1);
            tot = arena_take_t<uint64_t>(a, 1);
            scr = arena_take_t<uint64_t>(a, scan_scratch_words(nwords));
        }
        if (!ext || !gr || (groups && !list && (!flags || !wcnt || !woff || !tot || !scr))) {
            if (shrink()) continue;
            return ms_fail(MS_ERR_NOMEM, "arena exhausted (group output)");
        }
        const unsigned tgrid = unsigned(minu((cap + 255) / 256, persistent_grid(256, 8)));
        if (list) {
            k_group_list<<<tgrid, 256, 0, st>>>(t, sf, words + 1, list);
            k_group_rank<<<unsigned((groups + 31) / 32), 256, 0, st>>>(t, list, unsigned(groups), ext);
            MS_CUDA_TRY(cudaGetLastError());
        } else if (groups) {
            // first rows -> flags -> ranks
            MS_CUDA_TRY(cudaMemsetAsync(flags, 0, 4 * (nwords + 1), st));
            k_group_list<<<tgrid, 256, 0, st>>>(t, sf, words + 1, nullptr);
            k_group_flags<<<tgrid, 256, 0, st>>>(t, flags);
            k_popc_words<<<persistent_grid(256, 8), 256, 0, st>>>(flags, nwords, wcnt);
            MS_CUDA_TRY(cudaGetLastError());
            MS_CUDA_TRY(scan_exclusive<uint32_t>(wcnt, nwords, woff, tot, scr, st));
            k_group_extents<<<tgrid, 256, 0, st>>>(t, flags, woff, ext);
            MS_CUDA_TRY(cudaGetLastError());
        }
        if (nbt) {
            const unsigned grid = unsigned(minu((nbt + 7) / 8, persistent_grid(256, 3)));
            if (binary) {
                k_group_ids<true><<<grid, 256, 0, st>>>(gv, cv, t, nullptr, 0, gr, a->d_err);
            } else if (list && groups <= kGrpSmemGroups) {
                MS_CUDA_TRY(cudaFuncSetAttribute(k_group_ids<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 int(smem)));
                k_group_ids<false><<<grid, 256, smem, st>>>(gv, cv, t, list, unsigned(groups), gr, a->d_err);
            } else {
                k_group_ids<false><<<grid, 256, 0, st>>>(gv, cv, t, nullptr, 0, gr, a->d_err);
            }
            MS_CUDA_TRY(cudaGetLastError());
        }
        ReadBack end(a, st);
        const unsigned long long *h_scal = end.add(words + 2);
        rc = end.wait();
        if (rc) return rc;
        const uint64_t n_scal_groups = *h_scal;
        const uint64_t n_scal_rows = n - sf;
        rc = write_values(gr, n - n_scal_rows, n_scal_rows, gr_format, 0, out_gr, a, st);
        if (!rc) rc = write_values(ext, groups - n_scal_groups, n_scal_groups, ext_format, 0, out_ext, a, st);
        if (rc == MS_ERR_NOMEM && shrink()) continue;
        return rc;
    }
}

extern "C" int ms_gpu_agg_sum_grouped(const ms_col *gr, const ms_col *data, uint64_t n_groups, ms_col *out,
                                      ms_arena *a, void *stream) {
    if (!gr || !data || !out || !a) return ms_fail(MS_ERR_INVALID, "agg_sum_grouped: null argument");
    if (gr->count_values != data->count_values)
        return ms_fail(MS_ERR_INVALID, "agg_sum: inGrCol and inDataCol must contain the same number of data elements");
    cudaStream_t st = (cudaStream_t)stream;
    ColView gv, dv;
    int rc = view_or_decompress(gr, a, st, &gv);
    if (rc) return rc;
    rc = view_or_decompress(data, a, st, &dv);
    if (rc) return rc;
    uint64_t *res = arena_take_t<uint64_t>(a, n_groups + 1);
    if (!res) return ms_fail(MS_ERR_NOMEM, "arena exhausted (grouped sum)");
    MS_CUDA_TRY(cudaMemsetAsync(res, 0, 8 * (n_groups + 1), st));
    const uint64_t nbt = gv.nblocks_total();
    if (nbt && n_groups) {
        if (n_groups <= kSumSmemGroups) {
            unsigned copies = 1;
            const unsigned stride = unsigned(n_groups) | 1u;
            while (copies < 8 && 16ull * copies * stride <= kSumCopyBytes) copies <<= 1;
            // three CTAs of 256 threads per SM while their sums fit side by
            // side, else one of 768
            const size_t smem = 8ull * copies * stride;
            const bool wide = smem > 72 * 1024;
            const unsigned threads = wide ? 768 : 256;
            rc = allow_smem(k_grouped_sum, 8 * (kSumSmemGroups + 1));
            if (rc) return rc;
            const uint64_t per = threads / 32;
            const unsigned grid = unsigned(minu((nbt + per - 1) / per, persistent_grid(threads, wide ? 1 : 3)));
            k_grouped_sum<<<grid, threads, smem, st>>>(gv, dv, n_groups, copies, stride, (unsigned long long *)res,
                                                       a->d_err);
        } else {
            k_grouped_sum_many<<<unsigned(minu((nbt + 7) / 8, persistent_grid(256, 3))), 256, 12 * kSumSlots, st>>>(
                gv, dv, n_groups, (unsigned long long *)res, a->d_err);
        }
        MS_CUDA_TRY(cudaGetLastError());
    }
    rc = read_err(a, st);
    if (rc) return rc;
    *out = ms_col{};
    out->format = MS_FMT_UNCOMPR;
    out->count_values = n_groups;
    out->size_used_byte = 8 * n_groups;
    out->size_alloc_byte = 8 * (n_groups + 1);
    out->data = res;
    return MS_OK;
}

// join<ve, outL_f, outR_f, L_f, R_f>(L, R) (join.h:158-187,
// join_natural_equi_compr.h:116-300): (build position, probe position)
// pairs in probe order; the two outputs follow the write iterator model in
// their formats.
extern "C" int ms_gpu_natural_join(const ms_col *l, const ms_col *r, int out_l_format, unsigned out_l_bw,
                                   int out_r_format, unsigned out_r_bw, ms_col *out_l, ms_col *out_r, ms_arena *a,
                                   void *stream) {
    if (!l || !r || !out_l || !out_r || !a) return ms_fail(MS_ERR_INVALID, "natural_join: null argument");
    cudaStream_t st = (cudaStream_t)stream;
    ColView lv, rv;
    int rc = view_or_decompress(l, a, st, &lv);
    if (rc) return rc;
    rc = view_or_decompress(r, a, st, &rv);
    if (rc) return rc;
    unsigned long long *mm = arena_take_t<unsigned long long>(a, 3);
    if (!mm) return ms_fail(MS_ERR_NOMEM, "arena exhausted (natural_join)");
    const uint64_t nbl = lv.nblocks_total(), nl = l->count_values;
    uint64_t hmm[2] = {0, 0};
    if (nbl) {
        rc = key_range(lv, mm, hmm, hmm + 1, a, st);
        if (rc) return rc;
    }
    MS_CUDA_TRY(cudaMemsetAsync(mm + 2, 0xFF, 8, st));
    KeyMap m{};
    m.max_pos = mm + 2;
    if (nl && nl < 0xFFFFFFFFull && hmm[1] - hmm[0] < (uint64_t(1) << 24)) {
        m.lo = hmm[0];
        m.span = hmm[1] - hmm[0] + 1;
        const uint64_t words = (m.span + 31) / 32;
        m.dense = arena_take_t<uint32_t>(a, m.span);
        m.bits = arena_take_t<uint32_t>(a, words);
        if (!m.dense || !m.bits) return ms_fail(MS_ERR_NOMEM, "arena exhausted (natural_join array)");
        MS_CUDA_TRY(cudaMemsetAsync(m.dense, 0xFF, 4 * m.span, st));
        MS_CUDA_TRY(cudaMemsetAsync(m.bits, 0, 4 * words, st));
    } else {
        uint64_t cap = 16;
        while (cap < 2 * nl) cap <<= 1;
        m.keys = arena_take_t<unsigned long long>(a, cap);
        m.vals = arena_take_t<unsigned long long>(a, cap);
        if (!m.keys || !m.vals) return ms_fail(MS_ERR_NOMEM, "arena exhausted (natural_join table)");
        MS_CUDA_TRY(cudaMemsetAsync(m.keys, 0xFF, 8 * cap, st));
        MS_CUDA_TRY(cudaMemsetAsync(m.vals, 0xFF, 8 * cap, st));
        m.mask = cap - 1;
    }
    if (nbl) {
        k_build_map<<<grid_blocks(nbl), 256, 0, st>>>(lv, m, a->d_err);
        MS_CUDA_TRY(cudaGetLastError());
    }
    const uint64_t words = (m.span + 31) / 32;
    const bool smem = m.dense && smem_bitmap(words, rv.nblocks_total());
    uint64_t *pr, *pl, total, scal;
    // build positions of 32 bits unless the build side is longer
    auto join = [&](auto pos_type) -> int {
        using V = decltype(pos_type);
        if (smem) {
            int e = allow_smem(k_probe_map_bits<true, V>, 4 * kSmemBitmapWords);
            if (e) return e;
        }
        auto pass1 = [&](const MaskRun &run, V *side) {
            if (smem)
                k_probe_map_bits<true, V><<<mask_grid(run.nblk, kProbeWarps, 1), 32 * kProbeWarps, 4 * words, st>>>(
                    rv, m, run, side, a->d_err);
            else
                k_probe_map_bits<false, V><<<mask_grid(run.nblk, 8, 3), 256, 0, st>>>(rv, m, run, side, a->d_err);
        };
        return rows_by_mask<kRows | kVals, V>(rv, pass1, &pr, &pl, &total, &scal, a, st);
    };
    rc = nl < 0xFFFFFFFFull ? join(uint32_t(0)) : join(uint64_t(0));
    if (rc) return rc;
    rc = write_values(pl, total - scal, scal, out_l_format, out_l_bw, out_l, a, st);
    if (rc) return rc;
    return write_values(pr, total - scal, scal, out_r_format, out_r_bw, out_r, a, st);
}
