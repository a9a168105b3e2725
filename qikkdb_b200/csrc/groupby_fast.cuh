// The fast form of the fused filter + hash-aggregate pass, for calls of 16-byte aligned columns that hold a whole tile
// (the replacement of kernel_filter -> reconstructColKeep -> group_by_kernel,
// qikkDB/QueryEngine/GPUCore/GPUFilter.cuh:22-44, GPUReconstruct.cuh:272-355, GPUGroupBy.cuh:68-196, and of the
// multi-key kernel_group_by_multi_key, GPUGroupByMultiKey.cuh:156-259, for (int32, int32) keys).
//
// One persistent CTA per SM: a producer warp streams 2048-row tiles of the key, value and predicate columns into a
// ring of shared-memory stages with cp.async.bulk (TMA engine, mbarrier completion, evict-first L2 policy); 16
// consumer warps take the stages in order.  Warp w owns rows [128 w, 128 (w + 1)) of a tile and reads them as four
// 32-row segments (lane l: rows 32 j + l), so the predicate loads are conflict-free and the ballot of segment j lists
// its passing rows in row order.  The passing rows are then processed 32 at a time:
//   * the key's bucket is two slots whose key words are read with one 16-byte load;
//   * a hit updates the slot with 32-bit shared atomics only: a u32 count, a 64-bit sum kept as two u32 limbs (the
//     carry out of the low limb is read from the value the atomic returns) and min/max issued only when the value
//     improves on the slot's bound.  Integer sums wrap like the reference's 64-bit atomicAdd; float and double
//     values are added in fixed point (q = v * 2^F, F from the CTA's first tile and its row count, so that no sum
//     can overflow), exactly for float values; values outside that window take the FP64 global path;
//   * a table of few groups keeps up to 32 copies of every slot's state, one per lane, so that lanes of a warp that
//     meet on one key update different words (the copies are added up when the table is merged);
//   * a miss is appended to its partition's cell of the hash-partitioned spill area (gb_fspill_kernel aggregates
//     each partition in shared memory afterwards) or, without one, inserted into the global table.
// At the end every CTA merges its table into the global open-addressing table.
#pragma once

#include "groupby_agg.cuh"

namespace qdb {

constexpr int kFastWarps = 16;                      // consumer warps
constexpr int kFastThreads = (kFastWarps + 1) * 32; // + one producer warp
constexpr int kFastSeg = 4;                         // 32-row segments per warp and tile
constexpr int kFastR = 32 * kFastSeg;               // rows per warp and tile
constexpr int kFastT = kFastWarps * kFastR;         // rows per tile (2048)
constexpr int kMaxSpillBits = 13;                   // partitions the aggregation pass writes: at most 8192
constexpr int kMaxSpill2Bits = 6;                   // second-level partitions per first-level one: at most 64
// The NULL key's word in the shared tables and the spill (the global table has a slot of its own for it).  A real key
// with this word is never put there: it goes to the global table.
constexpr uint64_t kNullWord = kEmpty + 1;
constexpr int kTouchCap = 64;                       // queued keys per warp (FM_NULL)
// Buckets a key may be placed in where a table holds every group (a key that finds no place takes the global table for
// every row).
constexpr int kProbeBuckets = 64;
constexpr uint64_t kHashMul = 0x9E3779B97F4A7C15ull;

__device__ __forceinline__ uint32_t atoms_or(uint32_t a, uint32_t x) {
    uint32_t old;
    asm volatile("atom.shared.or.b32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(x) : "memory");
    return old;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t x) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ void lds128(uint32_t a, uint64_t& k0, uint64_t& k1) {
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(k0), "=l"(k1) : "r"(a) : "memory");
}

// Shared-window addresses of the bucketed table's arrays.  A bucket is two slots whose key words sit side by side
// (keys[2 b + j]); the slot's state lives in position-major arrays at index s = j NB + b, so that the states of
// different buckets' first positions fall in consecutive banks.
//
// A table of few groups keeps 2^rep_shift copies of every state (slot s, copy r at index (s << rep_shift) + r); lane l
// of every warp updates copy l mod 2^rep_shift and the merge adds the copies up.
struct FTab {
    uint32_t keys, cnt, l0, l1, l2, mn, mx;  // state arrays: the address of this lane's copy of slot 0
    uint32_t NB;
    uint32_t osh;                    // slot s's 4-byte state is at s << osh
};

template <typename VT>
__device__ __forceinline__ FTab ftab(unsigned char* sm, const AggArgs& a) {
    FTab t;
    const uint32_t r = threadIdx.x & ((1u << a.rep_shift) - 1u);
    t.keys = smem_u32(sm + a.so_keys);
    t.cnt = smem_u32(sm + a.so_cnt) + r * 4u;
    t.l0 = smem_u32(sm + a.so_l0) + r * 4u;
    t.l1 = smem_u32(sm + a.so_l1) + r * 4u;
    t.l2 = smem_u32(sm + a.so_l2) + r * 4u;
    t.mn = smem_u32(sm + a.so_mn) + r * static_cast<uint32_t>(sizeof(VT));
    t.mx = smem_u32(sm + a.so_mx) + r * static_cast<uint32_t>(sizeof(VT));
    t.NB = static_cast<uint32_t>(a.NB);
    t.osh = 2u + static_cast<uint32_t>(a.rep_shift);
    return t;
}

// Hash of a key word for the shared tables and the spill: one 64-bit multiply (Fibonacci hashing, Knuth TAOCP vol. 3,
// 6.4).  Its top bits pick the spill partition, the 32 bits below bit `shift` (32 - partition bits) the bucket (so
// a partition's rows spread over every bucket of the spill pass's table), and bits 32..46 the bit of the seen-once
// filter.  The global table hashes with the independent mix64.  Being linear it spreads dense and evenly spaced keys
// better than chance (no full buckets at half load, against 7-10 % with a mixing hash, which made the spill pass of
// 16.8M composite groups 4.2 instead of 3.8 ms), at the price of strides that it lines up: see ffar.
__device__ __forceinline__ uint64_t fhash(uint64_t kw) { return kw * kHashMul; }
__device__ __forceinline__ uint32_t fbucket(uint64_t m, int shift, uint32_t NB) {
    const uint32_t x = __funnelshift_rc(static_cast<uint32_t>(m), static_cast<uint32_t>(m >> 32), shift);
    return __umulhi(x, NB);
}

// Where a key whose home bucket is full goes: to the two buckets behind it, which the linear hash leaves emptier than
// chance, then to one from other bits of its hash, as home buckets that an unlucky stride of the keys lines up would also
// fill their neighbours.  The next bucket is looked into without a call; a key beyond it costs its warp a call in every
// step.  Both ends matter: with the far bucket first, 2^26 rows, half selected, over 300 float keys take 512 us (342 now),
// and 2^24 rows over 30,000 keys spaced by 0x9E3779B1, SUM/MIN/MAX/COUNT, 277 us in the spill pass (190 now); without it
// 10M rows over 20,000 keys spaced by 0x9E3779B97F4A7C15 take 763 us there.  Looking into two more buckets inline costs
// registers that the passes do not have (33M masked rows of doubles: 1317 instead of 1235 us).
__device__ __forceinline__ uint32_t fnext(uint32_t b, uint32_t NB) { return (b + 1u == NB) ? 0u : b + 1u; }
__device__ __forceinline__ uint32_t ffar(uint64_t m, uint32_t NB) {
    return __umulhi((static_cast<uint32_t>(m) ^ static_cast<uint32_t>(m >> 32)) * 0x9E3779B1u, NB);
}

// Looks kw up in bucket b: returns its slot or -1; empty: the bucket has a free position.
__device__ __forceinline__ int fprobe(const FTab& t, uint32_t b, uint64_t kw, bool& empty) {
    uint64_t k0, k1;
    lds128(t.keys + b * 16u, k0, k1);
    empty = (k0 == kEmpty) | (k1 == kEmpty);
    return (k0 == kw) ? static_cast<int>(b) : ((k1 == kw) ? static_cast<int>(t.NB + b) : -1);
}

// Finds or claims kw in bucket b, its two neighbours, the far one and those after it (nb buckets in all): a new key is
// claimed with a CAS on its key word.  full: bucket b is full and without kw.  Returns the slot or -1.
static __device__ __noinline__ int fclaim(const FTab t, uint32_t b, uint64_t kw, int nb, bool full) {
    uint32_t bb = full ? fnext(b, t.NB) : b;
    for (int k = full ? 1 : 0; k < nb; ++k) {
        if (k == 3) bb = ffar(fhash(kw), t.NB);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t ka = t.keys + (bb * 2u + j) * 8u;
            const uint64_t cur = lds64(ka);
            if (cur == kw) return static_cast<int>(j * t.NB + bb);
            if (cur == kEmpty) {
                const uint64_t prev = atoms_cas64(ka, kEmpty, kw);
                if (prev == kEmpty || prev == kw) return static_cast<int>(j * t.NB + bb);
            }
        }
        bb = fnext(bb, t.NB);
    }
    return -1;
}

// ---------------------------------------------------------------------------------------------
// 64-bit fixed-point sum addends.  A CTA that may add up to 2^hb - 1 values into one slot keeps every addend below
// 2^(63 - hb) in magnitude, so the slot's two's-complement sum cannot overflow.  emax is the largest binary exponent
// (|v| < 2^emax) of the CTA's first tile; values up to 2^(emax + 2) are kept.
//   float: q = m24 << sh with sh = biased exponent - sh0 in [0, min(30, 39 - hb)]: exact.  (The bound of 30 lets one widening
//   multiply shift and sign-extend; it narrows the window of spill items of fewer than 512 rows only, whose values below
//   2^-28 of the largest are added in FP64.)
//   double: q = round(v * 2^F) for |v| in [lo, hi): every kept value has at least 24 significant bits.
// FM_WIDE (calls with NULL masks or a row mask) keeps sums in 96 bits (three limbs), so that 64-bit addends need no
// headroom and the window is wide enough for columns that grow along their rows: values up to 2^(emax + 15) and down to
// 2^(emax - 24) are kept.  (With the 2^(emax + 2) of the 64-bit sums, 2^23 masked rows that grow 2^12-fold over 10 groups
// took 7.3 ms in FP64 atomics on ten words, 0.11 ms in the general pass.)
//   float: q = m24 << sh with sh in [0, 38]: exact.
//   double: q = round(v * 2^F) for |v| < 2^(emax + 2) and round(v * 2^(F - 13)) << 13 above, F = 61 - emax, less for CTAs
//   of 2^19 rows and more so that 2^hb values of 2^(emax + 15) fit 96 bits: 37 bits of the smallest kept value and more
//   of the others, 24 in CTAs of 2^32 rows.
// ---------------------------------------------------------------------------------------------
struct FixQ {
    int sh0 = 0;
    int shmax = 0;
    double scale = 1.0;  // 2^F
    double inv = 1.0;    // 2^-F
    double lo = 0.0;
    double hi = 0.0;
    double top = 0.0;        // FM_WIDE doubles: values in [hi, top) are added kWideShift bits up
};
constexpr int kWideShift = 13;

template <typename VT, bool WIDE>
__device__ __forceinline__ FixQ fixq(int emax, int hb) {
    FixQ f;
    if constexpr (WIDE && std::is_same<VT, float>::value) {
        f.shmax = 38;
        f.sh0 = max(1, min(254 - f.shmax, emax + 103));  // 2^(emax + 14) <= |v| < 2^(emax + 15) takes sh = 38
        f.inv = ldexp(1.0, f.sh0 - 150);
        return f;
    } else if constexpr (WIDE) {
        emax = max(-960, min(960, emax));
        const int F = 61 - emax - max(0, hb - 19);
        f.scale = ldexp(1.0, F);
        f.inv = ldexp(1.0, -F);
        f.lo = ldexp(1.0, emax - 24);
        f.hi = ldexp(1.0, emax + 2);
        f.top = ldexp(1.0, emax + 2 + kWideShift);
        return f;
    }
    emax = max(-900, min(900, emax));
    const int g = 2;
    f.shmax = max(0, min(30, 39 - hb));
    if constexpr (std::is_same<VT, float>::value) {
        // A value of exponent emax + g would take sh = shmax.  sh0 stays in [1, 254 - shmax], so the biased exponents
        // 0 (zero, subnormals) and 255 (Inf, NaN) always fall outside [sh0, sh0 + shmax].
        f.sh0 = max(1, min(254 - f.shmax, emax + 126 + g - f.shmax));
        f.scale = ldexp(1.0, 150 - f.sh0);         // q = v * 2^(150 - sh0)
        f.inv = ldexp(1.0, f.sh0 - 150);
    } else {
        const int F = 63 - hb - emax - g;          // |v| < 2^(emax + g) gives |q| < 2^(63 - hb)
        f.scale = ldexp(1.0, F);
        f.inv = ldexp(1.0, -F);
        f.hi = ldexp(1.0, emax + g);
        f.lo = ldexp(1.0, emax + g - f.shmax - 1);
    }
    return f;
}

template <typename VT, bool WIDE>
__device__ __forceinline__ long long addq(VT v, const FixQ& f, bool& ok) {
    if constexpr (std::is_same<VT, float>::value) {
        const uint32_t b = __float_as_uint(v);
        const uint32_t sh = ((b >> 23) & 0xffu) - static_cast<uint32_t>(f.sh0);  // below sh0: wraps to a large value
        const bool inw = sh <= static_cast<uint32_t>(f.shmax);
        ok = inw | ((b << 1) == 0u);  // zero is exact; subnormals, NaN and Inf take the FP64 path
        const int32_t sg = static_cast<int32_t>(b) >> 31;
        const int32_t m = static_cast<int32_t>(((b & 0x7fffffu) | 0x800000u) ^ static_cast<uint32_t>(sg)) - sg;
        if constexpr (WIDE) return static_cast<long long>(inw ? m : 0) << (sh & 63u);
        // one widening multiply shifts and sign-extends (fixq keeps sh at 30 or less)
        return static_cast<long long>(inw ? m : 0) * static_cast<long long>(static_cast<int32_t>(1u << (sh & 31u)));
    } else if constexpr (std::is_same<VT, double>::value) {
        const double m = fabs(v);
        ok = (m == 0.0) | ((m >= f.lo) & (m < (WIDE ? f.top : f.hi)));  // false for NaN and Inf
        const double down = WIDE && m >= f.hi ? 1.0 / (1 << kWideShift) : 1.0;  // update() shifts the addend back up
        return ok ? __double2ll_rn(v * down * f.scale) : 0ll;
    } else {
        ok = true;
        return static_cast<long long>(v);
    }
}

// Largest binary exponent of a finite non-zero value, INT_MIN otherwise (integers: INT_MIN).
template <typename VT>
__device__ __forceinline__ int fexp(VT v) { return value_exp<VT>(v); }

// ---------------------------------------------------------------------------------------------
// Table initialisation and merge into the global table.
// ---------------------------------------------------------------------------------------------
template <typename VT, bool WIDE>
__device__ __forceinline__ void ftab_init(unsigned char* sm, const AggArgs& a, int tid, int nthreads) {
    const int S = a.NB * 2;
    uint64_t* keys = reinterpret_cast<uint64_t*>(sm + a.so_keys);
    unsigned* cnt = reinterpret_cast<unsigned*>(sm + a.so_cnt);
    unsigned* l0 = reinterpret_cast<unsigned*>(sm + a.so_l0);
    unsigned* l1 = reinterpret_cast<unsigned*>(sm + a.so_l1);
    using MT = typename std::conditional<sizeof(VT) == 4, int, long long>::type;  // encoded min / max
    MT* mn = reinterpret_cast<MT*>(sm + a.so_mn);
    MT* mx = reinterpret_cast<MT*>(sm + a.so_mx);
    for (int i = tid; i < S; i += nthreads) keys[i] = kEmpty;
    const int E = S << a.rep_shift;
    for (int i = tid; i < E; i += nthreads) {
        cnt[i] = 0u;
        if (a.has_sum) {
            l0[i] = 0u;
            l1[i] = 0u;
            if (WIDE) reinterpret_cast<unsigned*>(sm + a.so_l2)[i] = 0u;
        }
        if (a.has_min) mn[i] = sizeof(VT) == 4 ? static_cast<MT>(INT_MAX) : static_cast<MT>(kMinInit64);
        if (a.has_max) mx[i] = sizeof(VT) == 4 ? static_cast<MT>(INT_MIN) : static_cast<MT>(kMaxInit64);
    }
}

// Merges every occupied slot into the global table (whole CTA).  Each thread takes U slots at a time and finds their
// global slots in lock-step rounds: a round issues the pending probe loads, or the claims (CAS) of keys that met an
// empty slot, of all U before it looks at any result, so their L2/DRAM round trips overlap.  A key still unresolved
// after a.flush_rounds rounds (a long probe run) finishes with the one-key search, which bounds the probe and reports
// a full table.

// SPILL: the table of a spill item, which has no copies of states and no NULL key.
template <typename VT, bool WIDE, bool SPILL = false>
__device__ __forceinline__ void ftab_flush(unsigned char* sm, const AggArgs& a, const FixQ& fq,
                                           unsigned long long* claims, bool null_seen = true) {
    constexpr bool V32 = sizeof(VT) == 4;
    constexpr bool VFLOAT = std::is_floating_point<VT>::value;
    const int S = a.NB * 2;
    const int W = a.L.W;
    const uint64_t* keys = reinterpret_cast<const uint64_t*>(sm + a.so_keys);
    const unsigned* cnt = reinterpret_cast<const unsigned*>(sm + a.so_cnt);
    const unsigned* l0 = reinterpret_cast<const unsigned*>(sm + a.so_l0);
    const unsigned* l1 = reinterpret_cast<const unsigned*>(sm + a.so_l1);
    const unsigned* l2 = reinterpret_cast<const unsigned*>(sm + a.so_l2);
    using MT = typename std::conditional<V32, int, long long>::type;
    const MT* smn = reinterpret_cast<const MT*>(sm + a.so_mn);
    const MT* smx = reinterpret_cast<const MT*>(sm + a.so_mx);
    const uint64_t mask = a.main.mask;
    constexpr int U = 4;
    for (int i0 = threadIdx.x; i0 < S; i0 += U * blockDim.x) {
        uint64_t key[U], pos[U], cur[U];
        uint64_t* g[U];
        bool pend[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int ki = i0 + u * blockDim.x;
            key[u] = (ki < S) ? keys[ki] : kEmpty;
            g[u] = nullptr;
            pend[u] = key[u] != kEmpty;
            if (!SPILL && a.null_keys && key[u] == kNullWord) {
                g[u] = null_seen ? g_special(a.main, W, 0, claims) : nullptr;
                pend[u] = false;
            }
            pos[u] = pend[u] ? home_slot(a.main, mix64(key[u])) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) cur[u] = pend[u] ? ld_volatile_u64(a.main.slots + pos[u] * W) : 0ull;
        for (int r = 0; r < a.flush_rounds && (pend[0] | pend[1] | pend[2] | pend[3]); ++r) {
            unsigned long long prev[U];
#pragma unroll
            for (int u = 0; u < U; ++u)  // claims of keys that met an empty slot, all issued before any is read
                prev[u] = (pend[u] && cur[u] == kEmpty)
                              ? atomicCAS(reinterpret_cast<unsigned long long*>(a.main.slots + pos[u] * W), kEmpty, key[u])
                              : cur[u];
            bool load[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                load[u] = false;
                if (!pend[u]) continue;
                if (prev[u] == key[u] || (cur[u] == kEmpty && prev[u] == kEmpty)) {
                    if (cur[u] == kEmpty && prev[u] == kEmpty) claim_counted(claims);
                    g[u] = a.main.slots + pos[u] * W;
                    pend[u] = false;
                } else {  // the slot holds another key: probe the next one
                    pos[u] = (pos[u] + 1) & mask;
                    load[u] = true;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (load[u]) cur[u] = ld_volatile_u64(a.main.slots + pos[u] * W);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (pend[u]) g[u] = g_find_from(a.main, W, key[u], pos[u], cur[u], a.counters, claims);
            if (!g[u]) continue;
            const int ki = i0 + u * blockDim.x;
            const int rep = SPILL ? 0 : a.rep_shift;
            const int i = ((ki & 1) * a.NB + (ki >> 1)) << rep;  // key index 2 b + j -> state j NB + b
            unsigned long long c = 0;
            uint64_t sum = 0;
            __int128 wide = 0;
            long long mn = V32 ? INT_MAX : LLONG_MAX, mx = V32 ? INT_MIN : LLONG_MIN;
#pragma unroll 1
            for (int k = 0; k < 1 << rep; ++k) {
                // lanes start at different copies, so the copies of neighbouring slots are read from different banks
                const int e = i + ((k + static_cast<int>(threadIdx.x)) & ((1 << rep) - 1));
                c += cnt[e];
                if (a.has_sum) {
                    const uint64_t lo = (static_cast<uint64_t>(l1[e]) << 32) | l0[e];
                    if (WIDE) wide += (static_cast<__int128>(static_cast<int32_t>(l2[e])) << 64) + static_cast<__int128>(lo);
                    else sum += lo;
                }
                if (a.has_min) mn = min(mn, static_cast<long long>(smn[e]));
                if (a.has_max) mx = max(mx, static_cast<long long>(smx[e]));
            }
            uint64_t sumbits = sum;
            if (a.has_sum && VFLOAT) {
                const double d = (WIDE ? limbs96_to_double(static_cast<unsigned>(wide), static_cast<unsigned>(wide >> 32),
                                                           static_cast<unsigned>(wide >> 64))
                                       : static_cast<double>(static_cast<long long>(sum))) * fq.inv;
                memcpy(&sumbits, &d, 8);
            }
            g_merge(g[u], a.L, a.has_sum, a.has_min, a.has_max, V32, VFLOAT, c, sumbits, mn, mx);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Rows of one step: two rows per lane (64 per warp), each row's table lookup, slot update and the fate of its miss.
// MODE bits: FM_SUM (a 64-bit sum), FM_MM (min and/or max), FM_VALS (a value column is read); without FM_VALS only
// the row count is kept.
// ---------------------------------------------------------------------------------------------
constexpr int FM_SUM = 1;
constexpr int FM_MM = 2;
constexpr int FM_VALS = 4;
constexpr int FM_KZ = 8;  // the key column is an AAFL-compressed block (single key, not DOUBLE)
constexpr int FM_NULL = 32;  // NULL masks (key, value, predicate) or a row mask; the predicate type is read at run time
constexpr int FM_WIDE = 64;  // 96-bit sums of floats and doubles
constexpr int FM_KMOD = 16;  // keys are replaced by key % m as they are read (single INT32 or INT64 key)

// K32: every key word is a 32-bit key's, so none equals kEmpty.
template <typename VT, int MODE, bool K32 = false>
struct FastWarp {
    static constexpr bool SUM = (MODE & FM_SUM) != 0;
    static constexpr bool MM = (MODE & FM_MM) != 0;
    static constexpr bool VALS = (MODE & FM_VALS) != 0;
    static constexpr bool NUL = (MODE & FM_NULL) != 0;
    static constexpr bool WIDE = (MODE & FM_WIDE) != 0;
    const AggArgs& a;
    FTab t;
    FixQ fq;
    unsigned long long* claims;
    int bshift = 32;       // bucket bits start at this bit of the hash
    int probe_b = 1;       // buckets a claim may visit
    bool fits = false;
    bool use_smem = true;  // probe the shared table at all
    bool spill_ok = false; // append misses to the spill area
    bool counting = true;  // count lookups and hits (until the warp has judged its hit rate)
    unsigned hits = 0, tries = 0;
    // Where a miss goes: partition q = (fhash(key) >> part_shift) & part_mask, appended to cell cell_base + q cell_mul
    // of spill_out (records of 16 bytes, or 8 for a count-only table) at the position its shared fill counter
    // sfill[q] hands out; a full cell sends the row to the global table.
    uint32_t sfill = 0;    // shared-window address of the per-partition fill counters
    uint32_t seen = 0;     // shared-window address of the seen-once filter (0: admit every key)
    unsigned cell_cap = 0;
    int part_shift = 64;
    uint32_t part_mask = 0;
    uint32_t cell_base = 0;
    uint32_t cell_mul = 0;
    uint64_t* spill_out = nullptr;
    // The NULL key's slot, claimed before the first row (FM_NULL with NULL keys), and the word that a NULL key sets.
    int null_slot = -1;
    uint32_t null_seen = 0;
    // Keys of rows with a NULL value that missed the table (they only have to exist in the global table), looked up 32
    // at a time.
    uint64_t* touch = nullptr;
    int touched = 0;

    __device__ __forceinline__ FastWarp(const AggArgs& args, const FTab& tab, const FixQ& f, unsigned long long* c)
        : a(args), t(tab), fq(f), claims(c) {}

    // One row into the global table; esc: kw is a real key although it is the NULL key's word; vn: its value is NULL.
    __device__ __forceinline__ void global_row(uint64_t kw, VT v, bool esc = false, bool vn = false) {
        uint64_t* slot = (kw == kEmpty) ? g_special(a.main, a.L.W, 1, claims)
                         : (a.null_keys && kw == kNullWord && !esc)
                             ? g_special(a.main, a.L.W, 0, claims)
                             : g_find(a.main, a.L.W, kw, mix64(kw), a.counters, claims);
        if (slot && !vn) {
            if (VALS) g_acc_row<VT>(slot, a, v);
            else g_count_row(slot, a.L);
        }
    }

    // Looks kw (hash m, home bucket b, full and without it) up in the next bucket it may be in: the slot or -1.
    __device__ __forceinline__ int look_on(uint64_t kw, uint64_t m, uint32_t b) const {
        bool empty;
        return fprobe(t, fnext(b, t.NB), kw, empty);
    }

    __device__ __forceinline__ void touch_queue(bool put, uint64_t kw, unsigned lane) {
        const unsigned b = __ballot_sync(0xffffffffu, put);
        if (b == 0u) return;
        if (put) touch[touched + __popc(b & ((1u << lane) - 1u))] = kw;
        touched += __popc(b);
        if (touched > kTouchCap - 32) touch_drain(lane, 32);
    }
    // Looks up the last `n` queued keys (at most 32).
    __device__ __forceinline__ void touch_drain(unsigned lane, int n) {
        __syncwarp();
        touched -= n;
        if (static_cast<int>(lane) < n) global_row(touch[touched + lane], VT{}, false, true);
        __syncwarp();
    }

    // Adds one row (its sum addend q, its value v) to slot s.
    __device__ __forceinline__ void update(uint32_t s, long long q, VT v) {
        const uint32_t o = s << t.osh;
        reds_add(t.cnt + o, 1u);
        if constexpr (SUM) {
            unsigned long long uq = static_cast<unsigned long long>(q);
            unsigned x2 = q < 0 ? 0xffffffffu : 0u;  // the addend's third word (FM_WIDE)
            if constexpr (WIDE && std::is_same<VT, double>::value) {
                if (fabs(v) >= fq.hi) {
                    x2 = static_cast<unsigned>(q >> (64 - kWideShift));
                    uq <<= kWideShift;
                }
            }
            const unsigned x0 = static_cast<unsigned>(uq);
            const unsigned old0 = atoms_add(t.l0 + o, x0);
            const unsigned c = (old0 + x0 < old0) ? 1u : 0u;
            if constexpr (WIDE) {
                const unsigned long long y1 = (uq >> 32) + c;
                const unsigned x1 = static_cast<unsigned>(y1);
                const unsigned old1 = atoms_add(t.l1 + o, x1);
                const unsigned y2 = x2 + static_cast<unsigned>(y1 >> 32) + ((old1 + x1 < old1) ? 1u : 0u);
                if (y2) reds_add(t.l2 + o, y2);
            } else {
                reds_add(t.l1 + o, static_cast<unsigned>(uq >> 32) + c);
            }
        }
        if constexpr (MM) {
            if constexpr (sizeof(VT) == 4) {
                const int32_t e = enc32(v);
                if (a.has_min && e < lds32(t.mn + o)) reds_min32(t.mn + o, e);
                if (a.has_max && e > lds32(t.mx + o)) reds_max32(t.mx + o, e);
            } else {
                const long long e = enc64(v);
                if (a.has_min && e < lds64s(t.mn + o * 2u)) reds_min64(t.mn + o * 2u, e);
                if (a.has_max && e > lds64s(t.mx + o * 2u)) reds_max64(t.mx + o * 2u, e);
            }
        }
    }

    // Stores a spilled row as one record (key word, value bits: a single 8- or 16-byte store) at position pos of its
    // partition's cell.
    __device__ __forceinline__ void spill_store(uint64_t kw, VT v, uint32_t p, unsigned pos) {
        const uint32_t idx = (cell_base + p * cell_mul) * cell_cap + pos;  // an area holds fewer than 2^31 records
        if constexpr (VALS) {
            uint64_t vb = 0;
            memcpy(&vb, &v, sizeof(VT));
            reinterpret_cast<ulonglong2*>(spill_out)[idx] = make_ulonglong2(kw, vb);
        } else {
            spill_out[idx] = kw;
        }
    }

    template <int U>
    __device__ __forceinline__ void rows(const bool (&act)[U], const uint64_t (&kw)[U], const VT (&v)[U], unsigned lane) {
        const bool no[U] = {};
        rows<U>(act, kw, v, no, no, lane);
    }

    // U rows per lane of a table that holds every group (no NULLs): the common row finds its key in its home bucket, and
    // everything else is worked out only in steps that hold such a row.  (In a spilling table, where most steps hold a
    // miss, that order costs a quarter more than rows(): 2.18 against 1.66 ms for 2^28 rows.)
    template <int U>
    __device__ __forceinline__ void rows_fit(const bool (&act)[U], const uint64_t (&kw)[U], const VT (&v)[U]) {
        long long q[U];
        bool look[U], hit[U], any_miss = false;
        uint64_t m[U];
        uint32_t b[U], slot[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            look[u] = true;
            q[u] = 0;
            if constexpr (SUM) q[u] = addq<VT, WIDE>(v[u], fq, look[u]);
            look[u] = look[u] & act[u];
            if constexpr (!K32) look[u] = look[u] & (kw[u] != kEmpty);
            m[u] = fhash(kw[u]);
            b[u] = fbucket(m[u], bshift, t.NB);
        }
        {
            uint64_t k0[U], k1[U];
#pragma unroll
            for (int u = 0; u < U; ++u) lds128(t.keys + b[u] * 16u, k0[u], k1[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool h0 = k0[u] == kw[u];
                hit[u] = look[u] & (h0 | (k1[u] == kw[u]));
                slot[u] = h0 ? b[u] : t.NB + b[u];
                any_miss |= act[u] & !hit[u];
            }
        }
        if (__any_sync(0xffffffffu, any_miss)) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (look[u] && !hit[u]) {
                    int s2 = look_on(kw[u], m[u], b[u]);  // a key whose home bucket is full
                    if (s2 < 0) s2 = fclaim(t, b[u], kw[u], probe_b, false);
                    hit[u] = s2 >= 0;
                    slot[u] = static_cast<uint32_t>(s2);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (act[u] && !hit[u]) global_row(kw[u], v[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (hit[u]) update(slot[u], q[u], v[u]);
    }

    // U rows per lane: (act[u], kw[u], v[u]) (FM_NULL: vn[u] its value is NULL, esc[u] kw[u] is a real key
    // that looks like the NULL key's word).  The rows' loads and arithmetic are independent, so
    // their latencies overlap; the rare paths (claims, next-bucket probes, misses) run under warp votes.
    template <int U>
    __device__ __forceinline__ void rows(const bool (&act)[U], const uint64_t (&kw)[U], const VT (&v)[U],
                                         const bool (&vn)[U], const bool (&esc)[U], unsigned lane) {
        long long q[U];
        bool inwin[U], look[U], hit[U], empty[U];
        uint64_t m[U], k0[U], k1[U];
        uint32_t b[U];
        int slot[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            inwin[u] = true;
            q[u] = 0;
            if constexpr (SUM) q[u] = addq<VT, WIDE>(v[u], fq, inwin[u]);
            if constexpr (NUL) inwin[u] = inwin[u] | vn[u];
            m[u] = fhash(kw[u]);
            look[u] = act[u] & (kw[u] != kEmpty) & inwin[u] & use_smem;
            if constexpr (NUL) look[u] = look[u] & (kw[u] != kNullWord);
            b[u] = fbucket(m[u], bshift, t.NB);
            k0[u] = k1[u] = kEmpty;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (look[u]) lds128(t.keys + b[u] * 16u, k0[u], k1[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool h0 = k0[u] == kw[u];
            hit[u] = look[u] & (h0 | (k1[u] == kw[u]));
            slot[u] = hit[u] ? static_cast<int>(h0 ? b[u] : t.NB + b[u]) : -1;
            empty[u] = (k0[u] == kEmpty) | (k1[u] == kEmpty);
            if constexpr (NUL) {
                // NULL keys never leave the table, also when it is not probed: they may be a large share of the rows.
                if (act[u] & (kw[u] == kNullWord) & !esc[u] & inwin[u]) {
                    slot[u] = null_slot;
                    hit[u] = true;
                    if (lds32(null_seen) == 0) sts32(null_seen, 1u);
                }
            }
        }
        if (fits) {
            // A table sized for every group places a key whose home bucket is full in the next one, or rarely in one after
            // it: look there before the claim path.
            bool nx[U], any_nx = false;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                nx[u] = look[u] & !hit[u] & !empty[u];
                any_nx |= nx[u];
            }
            if (__any_sync(0xffffffffu, any_nx)) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (nx[u]) {
                        const int s2 = look_on(kw[u], m[u], b[u]);
                        if (s2 >= 0) {
                            slot[u] = s2;
                            hit[u] = true;
                        }
                    }
                }
            }
        }
        // Claim path: a new key with room in its bucket or (a table sized for every group) any key not found so far.
        bool need[U], any_need = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            need[u] = look[u] & !hit[u] & (empty[u] | fits);
            any_need |= need[u];
        }
        if (__any_sync(0xffffffffu, any_need)) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                bool go = need[u];
                if (go && seen) {
                    // While a spilling table fills, a key is admitted on its second occurrence only, so that the
                    // slots go to keys that recur rather than to the first comers.
                    const uint32_t hb = static_cast<uint32_t>(m[u] >> 32) & 0x7fffu;
                    const uint32_t bit = 1u << (hb & 31u);
                    go = (atoms_or(seen + (hb >> 5) * 4u, bit) & bit) != 0u;
                }
                if (go) {
                    slot[u] = fclaim(t, b[u], kw[u], fits ? probe_b : 1, !empty[u]);
                    hit[u] = slot[u] >= 0;
                }
            }
        }
        if (counting) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                tries += look[u] ? 1u : 0u;
                hits += hit[u] ? 1u : 0u;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (hit[u] && !(NUL && vn[u])) update(static_cast<uint32_t>(slot[u]), q[u], v[u]);
        bool miss[U], any_miss = false;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            miss[u] = act[u] & !hit[u];
            any_miss |= miss[u];
        }
        if (__any_sync(0xffffffffu, any_miss)) {
            // All rows' spill positions are claimed before any record is stored, so the shared-atomic round
            // trips overlap; rows that cannot spill (or whose cell is full) go to the global table.
            bool sp[U];
            unsigned pos[U];
            uint32_t part[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                sp[u] = miss[u] & spill_ok & (kw[u] != kEmpty) & inwin[u];
                if constexpr (NUL) sp[u] = sp[u] & !vn[u] & !esc[u];
                part[u] = (sp[u] && part_shift < 64) ? static_cast<uint32_t>(m[u] >> part_shift) & part_mask : 0u;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) pos[u] = sp[u] ? atoms_add(sfill + part[u] * 4u, 1u) : 0u;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (sp[u] && pos[u] < cell_cap) {
                    spill_store(kw[u], v[u], part[u], pos[u]);
                } else if (NUL ? (miss[u] && (!vn[u] || esc[u] || kw[u] == kEmpty)) : miss[u]) {
                    global_row(kw[u], v[u], NUL && esc[u], NUL && vn[u]);
                }
            }
            if constexpr (NUL) {
#pragma unroll
                for (int u = 0; u < U; ++u) touch_queue(miss[u] & vn[u] & !esc[u] & (kw[u] != kEmpty), kw[u], lane);
            }
        }
    }
};

// Key of row R of an AAFL-compressed key column (the block layout of qikkDB's GPUCompression.cu / feathergpu AAFL):
// rows come in groups of 32 W (W = bits of the key type); row R is lane R % 32, value i = (R % 32W) / 32 of its group,
// and occupies bits [i b, (i + 1) b) of the lane's stream, whose word k is words[pos[g] + lane + 32 k], least
// significant bit first.  Lanes of a warp that hold consecutive rows read consecutive words.  A word index past the
// packed words (a malformed block) latches QDB_ERR_INVALID and yields the offset.
template <typename KT>
__device__ __forceinline__ KT kz_key(const AggArgs& a, int64_t R) {
    using WT = typename std::conditional<sizeof(KT) == 8, unsigned long long, unsigned int>::type;
    constexpr int W = sizeof(KT) * 8;
    const int64_t g = R / (32 * W);
    const int i = static_cast<int>((R % (32 * W)) >> 5);
    const int l = static_cast<int>(R & 31);
    const int b = a.kz_bits[g];
    WT x = 0;
    if (b) {
        const int o = i * b;
        const int k = o / W;
        const int p = o % W;
        const int64_t i0 = static_cast<int64_t>(a.kz_pos[g]) + l + 32 * k;
        const bool two = p + b > W;
        if (i0 >= 0 && i0 + (two ? 32 : 0) < a.kz_len) {
            const WT* w = static_cast<const WT*>(a.kz_words);
            x = w[i0] >> p;
            if (two) x |= w[i0 + 32] << (W - p);
            if (b < W) x &= (WT(1) << b) - WT(1);
        } else {
            atomicExch(reinterpret_cast<int*>(&a.counters[1]), static_cast<int>(QDB_ERR_INVALID));
        }
    }
    const WT v = static_cast<WT>(x + static_cast<WT>(a.kz_off));
    KT out;
    memcpy(&out, &v, sizeof(KT));
    return out;
}

// Compressed keys in the ring: stage s's key region holds the tile's groups (one of 64-bit words, two of 32-bit),
// group gi at byte gi kzSlot<KT>() of the region, each copied from the 16-byte boundary at or below its first word:
// the words start `lead` bytes into the slot.  kzb[4 s + 2 gi] is the group's bit length, kzb[4 s + 2 gi + 1] its lead.
template <typename KT>
constexpr uint32_t kzSlot() { return 32u * sizeof(KT) * 8u * sizeof(KT) + 32u; }
template <typename KT>
constexpr uint32_t kzStage() { return static_cast<uint32_t>(kFastT) * sizeof(KT) + 64u; }

template <typename KT>
__device__ __forceinline__ KT kz_ring(const unsigned char* keys, const uint8_t* kzb, int g, uint64_t off) {
    using WT = typename std::conditional<sizeof(KT) == 8, unsigned long long, unsigned int>::type;
    constexpr int W = sizeof(KT) * 8;
    constexpr int GW = 32 * W;
    const int s = g / kFastT;
    const int r = g % kFastT;
    const int gi = r / GW;
    const int i = (r % GW) >> 5;
    const int l = r & 31;
    const int b = kzb[4 * s + 2 * gi];
    WT x = 0;
    if (b) {
        const WT* w = reinterpret_cast<const WT*>(keys + static_cast<size_t>(s) * kzStage<KT>() + gi * kzSlot<KT>() +
                                                  kzb[4 * s + 2 * gi + 1]) + l;
        const int o = i * b;
        const int k = o / W;
        const int p = o % W;
        x = w[32 * k] >> p;
        if (p + b > W) x |= w[32 * (k + 1)] << (W - p);
        if (b < W) x &= (WT(1) << b) - WT(1);
    }
    const WT v = static_cast<WT>(x + static_cast<WT>(off));
    KT out;
    memcpy(&out, &v, sizeof(KT));
    return out;
}

// ---------------------------------------------------------------------------------------------
// The aggregation kernel.  KT: key column type; COMP: composite (int32, int32) key; VT: value type (int32_t for a
// count-only table); PT: predicate column type or NoPred; MODE: FM_* bits.
//
// The ring holds NS stages column by column: column c of stage s, row i is at so_stage + off_c + (s T + i) * size_c,
// so a list entry g = s T + i addresses a row of any stage.  With three or more stages, the passing rows a warp has not
// processed when a tile ends (fewer than 64) stay in its list and its hold on that stage continues until the next
// tile's first step has taken them, so every step but the last has 64 rows.
// ---------------------------------------------------------------------------------------------
constexpr int kListCap = 192;  // list entries per warp: fewer than 64 carried plus a tile's 128

// The predicate interval test in the column's type.
template <typename T>
__device__ __forceinline__ bool pred_pass(const PredInterval& pi, T x) {
    return ((x >= from_bits<T>(pi.lo)) & (x <= from_bits<T>(pi.hi))) != (pi.invert != 0);
}
__host__ __device__ __forceinline__ int pred_size(int32_t t) {
    return (t == QDB_INT32 || t == QDB_FLOAT) ? 4 : ((t == QDB_INT64 || t == QDB_DOUBLE) ? 8 : 0);
}

// A key's C++ remainder by the call's modulus (the fused key % m variant).
template <typename KT>
__device__ __forceinline__ KT kmod_key(const AggArgs& a, KT k) {
    return static_cast<KT>(mod_signed(static_cast<int64_t>(k), a.km_d, a.km_m, a.km_s1, a.km_s2));
}

template <typename KT, bool COMP, typename VT, typename PT, int MODE>
__global__ void __launch_bounds__(kFastThreads, 1) gb_fast_kernel(const AggArgs a) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ unsigned long long s_claims;
    __shared__ int s_emax;
    __shared__ int s_null_slot;
    __shared__ unsigned s_null_seen;
    constexpr bool HAS_PRED = !std::is_same<PT, NoPred>::value;
    constexpr bool VFLOAT = std::is_floating_point<VT>::value;
    constexpr bool VALS = (MODE & FM_VALS) != 0;
    constexpr bool KZ = !COMP && (MODE & FM_KZ) != 0;
    constexpr bool KMOD = !COMP && !KZ && (MODE & FM_KMOD) != 0 && std::is_integral<KT>::value;
    constexpr bool NUL = !COMP && (MODE & FM_NULL) != 0;
    constexpr bool WIDE = (MODE & FM_WIDE) != 0;
    constexpr bool LIST = HAS_PRED || NUL;  // rows are filtered into the warp's list
    // Rows a lane takes per step: a warp's whole slice of a tile where every row passes and no values are read, else two:
    // four rows with values do not fit the 96 registers (2^24 rows over 3000 groups, SUM of double, int32 keys: 191 us with
    // four, 159 with two; over 30,000 groups, SUM/MIN/MAX/COUNT of int32, int64 keys: 344 and 284.  Tables of wide rows that
    // hold every group would be 10 to 15 % faster with four, but their code beside the other costs both its registers).
    constexpr int U = LIST || VALS ? 2 : kFastSeg;
    using PL = typename std::conditional<HAS_PRED, PT, int32_t>::type;
    constexpr int PW = sizeof(PL);

    const FTab tab = ftab<VT>(sm, a);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(sm + a.so_bar);
    uint64_t* empty_bar = full_bar + a.NS;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const bool spill_on = a.spill_keys != nullptr;
    const int parts = spill_on ? (1 << a.spill_bits) : 0;
    unsigned* sfill = reinterpret_cast<unsigned*>(sm + a.so_spill);
    unsigned char* ring = sm + a.so_stage;
    const StageLayout& sl = a.sl;

    ftab_init<VT, WIDE>(sm, a, threadIdx.x, blockDim.x);
    if (spill_on) {
        for (int i = threadIdx.x; i < parts + kSeenWords; i += blockDim.x) sfill[i] = 0u;
        if (blockIdx.x == 0 && threadIdx.x == 0) a.spill_fill[static_cast<int64_t>(parts) * a.spill_ctas] = 0u;  // spill-pass work counter
    }
    if (threadIdx.x == 0) {
        s_claims = 0;
        s_emax = INT_MIN;
        s_null_slot = -1;
        s_null_seen = 0u;
        for (int s = 0; s < a.NS; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], kFastWarps);
        }
        mbar_fence_init();
    }
    __syncthreads();
    if constexpr (NUL) {
        if (a.null_keys && threadIdx.x == 0)  // an empty table always has room in the home bucket
            s_null_slot = fclaim(tab, fbucket(fhash(kNullWord), 32, tab.NB), kNullWord, 1, false);
        __syncthreads();
    }

    const int64_t my_tiles =
        (a.tiles > static_cast<int64_t>(blockIdx.x)) ? (a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    // Headroom of the fixed-point sums: a slot of this CTA receives fewer than 2^hb values.
    const int hb = max(1, 64 - __clzll(static_cast<long long>(my_tiles * kFastT)));
    FixQ fq;

    if (warp == kFastWarps) {
        // ---------------- producer warp: one elected lane issues the bulk copies ----------------
        if (lane == 0) {
            const uint64_t pol = l2_evict_first_policy();
            int64_t q = 0;
            int s = 0;
            uint32_t ph = 0;
            uint32_t tx = static_cast<uint32_t>(kFastT) * sizeof(KT) * ((COMP ? 2 : 1) - (KZ ? 1 : 0));
            if (VALS) tx += static_cast<uint32_t>(kFastT) * sizeof(VT);
            if (HAS_PRED) tx += static_cast<uint32_t>(kFastT) * PW;
            constexpr uint32_t NB8 = kFastT / 8;  // bytes of a tile's null words
            const uint32_t rpw = NUL ? static_cast<uint32_t>(pred_size(a.ptype)) : 0u;
            if constexpr (NUL) {
                tx += static_cast<uint32_t>(kFastT) * rpw;
                if (a.knull0) tx += NB8;
                if (a.vnull) tx += NB8;
                if (a.pnull) tx += NB8;
                if (a.mask) tx += kFastT;
            }
            for (; q < my_tiles; ++q) {
                const int64_t tile = blockIdx.x + q * static_cast<int64_t>(gridDim.x);
                if (tile >= a.full_tiles) break;  // the partial last tile is read directly
                if (q >= a.NS && !mbar_wait(&empty_bar[s], ph ^ 1u, a.counters)) break;
                const int64_t r0 = tile * kFastT;
                const size_t so = static_cast<size_t>(s) * kFastT;
                // Compressed keys: the tile's groups (one of 64-bit words, two of 32-bit) arrive as their packed words,
                // each copied from the 16-byte boundary at or below its first word through the 16-byte chunk that holds
                // its last (a chunk that holds a byte of the block lies in a page the block uses).
                constexpr int KZ_GW = 32 * static_cast<int>(sizeof(KT)) * 8;
                constexpr int KZ_NG = COMP ? 1 : kFastT / KZ_GW;
                uint32_t kz_bytes[2] = {0u, 0u};
                uint64_t kz_src[2] = {0ull, 0ull};
                if constexpr (KZ) {
                    uint8_t* kzb = reinterpret_cast<uint8_t*>(sm + a.so_bar + 96) + 4 * s;
#pragma unroll
                    for (int gi = 0; gi < KZ_NG; ++gi) {
                        const int64_t g = tile * KZ_NG + gi;
                        int b = a.kz_bits[g];
                        const uint64_t pos = a.kz_pos[g];
                        const uint64_t words = 32ull * static_cast<uint64_t>(b);
                        if (b > static_cast<int>(sizeof(KT)) * 8 || pos + words > static_cast<uint64_t>(a.kz_len)) {
                            if (b) atomicExch(reinterpret_cast<int*>(&a.counters[1]), static_cast<int>(QDB_ERR_INVALID));
                            b = 0;
                        }
                        const uint64_t src = reinterpret_cast<uint64_t>(a.kz_words) + pos * sizeof(KT);
                        const uint32_t lead = static_cast<uint32_t>(src & 15u);
                        kzb[2 * gi] = static_cast<uint8_t>(b);
                        kzb[2 * gi + 1] = static_cast<uint8_t>(lead);
                        kz_bytes[gi] = b ? ((lead + static_cast<uint32_t>(words * sizeof(KT)) + 15u) & ~15u) : 0u;
                        kz_src[gi] = src - lead;
                    }
                }
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(&full_bar[s], tx + kz_bytes[0] + kz_bytes[1]);
#pragma unroll
                for (int gi = 0; gi < KZ_NG; ++gi)
                    if (kz_bytes[gi])
                        bulk_g2s(ring + sl.key0 + static_cast<size_t>(s) * kzStage<KT>() + gi * kzSlot<KT>(),
                                 reinterpret_cast<const void*>(kz_src[gi]), kz_bytes[gi], &full_bar[s], pol);
                if constexpr (!KZ) bulk_g2s(ring + sl.key0 + so * sizeof(KT), static_cast<const KT*>(a.key0) + r0, kFastT * sizeof(KT), &full_bar[s], pol);
                if (COMP) bulk_g2s(ring + sl.key1 + so * sizeof(KT), static_cast<const KT*>(a.key1) + r0, kFastT * sizeof(KT), &full_bar[s], pol);
                if (VALS) bulk_g2s(ring + sl.val + so * sizeof(VT), static_cast<const VT*>(a.vals) + r0, kFastT * sizeof(VT), &full_bar[s], pol);
                if (HAS_PRED) bulk_g2s(ring + sl.pred + so * PW, static_cast<const PL*>(a.pcol) + r0, kFastT * PW, &full_bar[s], pol);
                if constexpr (NUL) {
                    const size_t sn = static_cast<size_t>(s) * NB8;
                    const int64_t w0 = r0 / 64;
                    if (rpw) bulk_g2s(ring + sl.pred + so * rpw, static_cast<const unsigned char*>(a.pcol) + r0 * rpw, kFastT * rpw, &full_bar[s], pol);
                    if (a.knull0) bulk_g2s(ring + sl.knull0 + sn, a.knull0 + w0, NB8, &full_bar[s], pol);
                    if (a.vnull) bulk_g2s(ring + sl.vnull + sn, a.vnull + w0, NB8, &full_bar[s], pol);
                    if (a.pnull) bulk_g2s(ring + sl.pnull + sn, a.pnull + w0, NB8, &full_bar[s], pol);
                    if (a.mask) bulk_g2s(ring + sl.mask + so, a.mask + r0, kFastT, &full_bar[s], pol);
                }
                if (++s == a.NS) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // Drain: every issued stage must have been consumed (so no copy is still in flight) before exit.
            for (int64_t d = (q > a.NS ? q - a.NS : 0); d < q; ++d) {
                const int sd = static_cast<int>(d % a.NS);
                if (!mbar_wait(&empty_bar[sd], static_cast<uint32_t>((d / a.NS) & 1), a.counters)) break;
            }
        }
    } else {
        // ---------------- consumer warps ----------------
        const PL plo = HAS_PRED ? from_bits<PL>(a.pi.lo) : PL{};
        const PL phi = HAS_PRED ? from_bits<PL>(a.pi.hi) : PL{};
        const bool pinv = a.pi.invert != 0;
        uint16_t* list = reinterpret_cast<uint16_t*>(sm + a.so_list) + warp * kListCap;
        const uint32_t lt_mask = (1u << lane) - 1u;
        const KT* rk0 = reinterpret_cast<const KT*>(ring + sl.key0);
        const KT* rk1 = reinterpret_cast<const KT*>(ring + sl.key1);
        const VT* rv = reinterpret_cast<const VT*>(ring + sl.val);
        const PL* rp = reinterpret_cast<const PL*>(ring + sl.pred);

        // Fixed-point scale of float sums: the largest exponent of this CTA's first tile of values.
        if (VFLOAT && (MODE & FM_SUM) && my_tiles > 0) {
            const int64_t tile = blockIdx.x;
            const bool staged = tile < a.full_tiles;
            bool ok = true;
            if (staged) ok = mbar_wait(&full_bar[0], 0u, a.counters);
            int e = INT_MIN;
            if (ok) {
                for (int j = lane; j < kFastR; j += 32) {
                    const int i = warp * kFastR + j;
                    const int64_t r = tile * kFastT + i;
                    if (r < a.n && !(NUL && null_bit(a.vnull, r)))
                        e = max(e, fexp<VT>(staged ? rv[i] : static_cast<const VT*>(a.vals)[r]));
                }
            }
            e = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0 && e != INT_MIN) atomicMax(&s_emax, e);
        }
        asm volatile("bar.sync 1, %0;" ::"r"(kFastWarps * 32) : "memory");
        fq = fixq<VT, WIDE>(s_emax == INT_MIN ? 0 : s_emax, hb);

        FastWarp<VT, MODE> fw(a, tab, fq, &s_claims);
        fw.bshift = 32;
        fw.fits = a.fits != 0;
        fw.counting = !fw.fits;
        fw.probe_b = a.probe_b;
        fw.spill_ok = spill_on;
        if (spill_on) {
            fw.sfill = smem_u32(sfill);
            fw.seen = smem_u32(sfill + parts);
            fw.cell_cap = static_cast<unsigned>(a.spill_cell);
            fw.part_shift = 64 - a.spill_bits;
            fw.part_mask = static_cast<uint32_t>(parts - 1);
            fw.cell_base = blockIdx.x;
            fw.cell_mul = static_cast<uint32_t>(a.spill_ctas);
            fw.spill_out = a.spill_keys;
        }
        auto pass = [&](PL x) -> bool { return ((x >= plo) & (x <= phi)) != pinv; };
        if constexpr (NUL) {
            fw.null_slot = s_null_slot;
            fw.null_seen = smem_u32(&s_null_seen);
        }
        if constexpr (NUL) fw.touch = reinterpret_cast<uint64_t*>(sm + a.so_touch) + warp * kTouchCap;
        // Null bit of the staged row g (stage s, row i at g = s T + i).
        auto ring_bit = [&](int32_t off, int g) -> bool {
            return off >= 0 && ((reinterpret_cast<const uint32_t*>(ring + off)[g >> 5] >> (g & 31)) & 1u);
        };
        // FM_NULL's filter: the predicate in its own type, its NULLs and the row mask.
        auto pass_any = [&](const void* col, int64_t i) -> bool {
            switch (a.ptype) {
                case QDB_INT32: return pred_pass<int32_t>(a.pi, static_cast<const int32_t*>(col)[i]);
                case QDB_INT64: return pred_pass<int64_t>(a.pi, static_cast<const int64_t*>(col)[i]);
                case QDB_FLOAT: return pred_pass<float>(a.pi, static_cast<const float*>(col)[i]);
                case QDB_DOUBLE: return pred_pass<double>(a.pi, static_cast<const double*>(col)[i]);
                default: return true;
            }
        };
        const uint8_t* kzb = reinterpret_cast<const uint8_t*>(sm + a.so_bar + 96);
        auto ring_row = [&](int g, uint64_t& kw, VT& v, bool& vn, bool& esc) {
            vn = esc = false;
            if constexpr (NUL) {
                const bool kn = ring_bit(sl.knull0, g);
                kw = kn ? kNullWord : key_word(rk0[g]);
                esc = !kn & (kw == kNullWord);
                vn = ring_bit(sl.vnull, g);
            } else if constexpr (COMP) kw = composite_word(static_cast<int32_t>(rk0[g]), static_cast<int32_t>(rk1[g]));
            else if constexpr (KZ) kw = key_word(kz_ring<KT>(ring + sl.key0, kzb, g, a.kz_off));
            else if constexpr (KMOD) kw = key_word(kmod_key<KT>(a, rk0[g]));  // of passing rows only
            else kw = key_word(rk0[g]);
            if constexpr (VALS) v = rv[g];
            else v = VT{};
        };
        // Steps over list entries [e0, e1): full steps, and the remainder when `flush`.  Returns the entries taken.
        const bool listed = LIST && (HAS_PRED || a.ptype || a.mask || a.pnull);  // FM_NULL without a filter: every row passes
        auto steps = [&](int total, bool flush, int g0) -> int {
            int e0 = 0;
            for (; e0 + 32 * U <= total || (flush && e0 < total); e0 += 32 * U) {
                bool act[U], vn[U], esc[U];
                uint64_t kw[U];
                VT v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int e = e0 + 32 * u + lane;
                    act[u] = e < total;
                    int g;
                    if (listed) g = list[act[u] ? e : e0];
                    else g = g0 + (act[u] ? e : e0);
                    ring_row(g, kw[u], v[u], vn[u], esc[u]);
                }
                fw.template rows<U>(act, kw, v, vn, esc, static_cast<unsigned>(lane));
            }
            return e0 < total ? e0 : total;
        };

        int s = 0;
        uint32_t ph = 0;
        int lc = 0;     // entries carried at the front of the list
        int held = -1;  // the stage those entries live in
        const bool carry = a.NS >= 3;
        int64_t tile = blockIdx.x;
        for (int64_t q = 0; q < my_tiles; ++q, tile += gridDim.x) {
            const bool staged = tile < a.full_tiles;
            if (!staged) {
                // The last, partial tile of the input: read directly from HBM, one step per 64 rows.
                const int64_t base = tile * kFastT;
                const int64_t lim = a.n - base;
                const int w0 = warp * kFastR;
                const KT* k0p = static_cast<const KT*>(a.key0) + base;
                const KT* k1p = static_cast<const KT*>(a.key1) + base;
                const VT* vp = static_cast<const VT*>(a.vals) + base;
                int count = 0;
                if constexpr (NUL) {
#pragma unroll
                    for (int j = 0; j < kFastSeg; ++j) {
                        const int i = w0 + 32 * j + lane;
                        const int64_t r = base + i;
                        const bool keep = i < lim && !null_bit(a.pnull, r) && (!a.mask || a.mask[r]) && pass_any(a.pcol, r);
                        const uint32_t bj = __ballot_sync(0xffffffffu, keep);
                        if (keep) list[count + __popc(bj & lt_mask)] = static_cast<uint16_t>(i);
                        count += __popc(bj);
                    }
                } else if constexpr (HAS_PRED) {
                    const PL* pp = static_cast<const PL*>(a.pcol) + base;
#pragma unroll
                    for (int j = 0; j < kFastSeg; ++j) {
                        const int i = w0 + 32 * j + lane;
                        const bool keep = i < lim && pass(pp[i]);
                        const uint32_t bj = __ballot_sync(0xffffffffu, keep);
                        if (keep) list[count + __popc(bj & lt_mask)] = static_cast<uint16_t>(i);
                        count += __popc(bj);
                    }
                } else {
                    count = static_cast<int>(lim - w0 < 0 ? 0 : (lim - w0 > kFastR ? kFastR : lim - w0));
                }
                __syncwarp();
                for (int e0 = 0; e0 < count; e0 += 32 * U) {
                    bool act[U], vn[U] = {}, esc[U] = {};
                    uint64_t kw[U];
                    VT v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int e = e0 + 32 * u + lane;
                        act[u] = e < count;
                        const int i = LIST ? list[act[u] ? e : e0] : w0 + (act[u] ? e : e0);
                        if constexpr (NUL) {
                            const bool kn = null_bit(a.knull0, base + i);
                            kw[u] = kn ? kNullWord : key_word(k0p[i]);
                            esc[u] = !kn & (kw[u] == kNullWord);
                            vn[u] = null_bit(a.vnull, base + i);
                        } else if constexpr (COMP) kw[u] = composite_word(static_cast<int32_t>(k0p[i]), static_cast<int32_t>(k1p[i]));
                        else if constexpr (KZ) kw[u] = key_word(kz_key<KT>(a, base + i));
                        else if constexpr (KMOD) kw[u] = key_word(kmod_key<KT>(a, k0p[i]));
                        else kw[u] = key_word(k0p[i]);
                        if constexpr (VALS) v[u] = vp[i];
                        else v[u] = VT{};
                    }
                    fw.template rows<U>(act, kw, v, vn, esc, static_cast<unsigned>(lane));
                }
                __syncwarp();
                continue;
            }
            if (!mbar_wait(&full_bar[s], ph, a.counters)) break;
            const bool full = (q & 127) == 0 && __any_sync(0xffffffffu, table_full(a.counters));
            // The next tile of this CTA is staged too: rows left over may wait for it.
            const bool keep_going = carry && !full && q + 1 < my_tiles && tile + gridDim.x < a.full_tiles;
            const int g0 = s * kFastT + warp * kFastR;  // ring index of the warp's first row in this stage
            int total = lc;
            if (!full) {
                if (NUL && !listed) {
                    total = kFastR;
                } else if constexpr (NUL) {
#pragma unroll
                    for (int j = 0; j < kFastSeg; ++j) {
                        const int g = g0 + 32 * j + lane;
                        const bool keep = !ring_bit(sl.pnull, g) && (sl.mask < 0 || ring[sl.mask + g]) && pass_any(ring + sl.pred, g);
                        const uint32_t bj = __ballot_sync(0xffffffffu, keep);
                        if (keep) list[total + __popc(bj & lt_mask)] = static_cast<uint16_t>(g);
                        total += __popc(bj);
                    }
                } else if constexpr (HAS_PRED) {
                    // Filter: segment j of the warp's slice is rows 32 j + lane; its ballot lists the passing rows in
                    // row order behind the carried entries.
#pragma unroll
                    for (int j = 0; j < kFastSeg; ++j) {
                        const int g = g0 + 32 * j + lane;
                        const bool keep = pass(rp[g]);
                        const uint32_t bj = __ballot_sync(0xffffffffu, keep);
                        if (keep) list[total + __popc(bj & lt_mask)] = static_cast<uint16_t>(g);
                        total += __popc(bj);
                    }
                } else {
                    total = kFastR;
                }
                __syncwarp();
            }
            int taken = full ? total : steps(total, !keep_going, g0);
            if (held >= 0 && taken == 0) taken = steps(total, true, g0);  // never hold two stages into the next tile
            __syncwarp();
            if (held >= 0 && lane == 0) mbar_arrive(&empty_bar[held]);  // its rows were the first lc entries
            held = -1;
            const int rem = total - taken;
            if (rem > 0) {
                // Move the leftover entries to the front (source at 64 or beyond, so the ranges do not overlap).
                const uint16_t t0 = lane < rem ? list[taken + lane] : 0;
                const uint16_t t1 = lane + 32 < rem ? list[taken + 32 + lane] : 0;
                __syncwarp();
                if (lane < rem) list[lane] = t0;
                if (lane + 32 < rem) list[32 + lane] = t1;
                __syncwarp();
                held = s;
            } else if (lane == 0) {
                mbar_arrive(&empty_bar[s]);
            }
            lc = rem;
            if (++s == a.NS) {
                s = 0;
                ph ^= 1u;
            }
            // After the table's fill phase a warp judges its hit rate: below 1/8 (keys spread evenly over many more
            // groups than the table holds) it stops probing the table and sends every row to the spill, which the
            // spill pass aggregates partition by partition in shared memory.
            if (q + 1 == kCountTile) fw.hits = fw.tries = 0;
            if (q == kDecideTile && fw.use_smem && fw.counting) {
                const unsigned h = __reduce_add_sync(0xffffffffu, fw.hits);
                const unsigned t = __reduce_add_sync(0xffffffffu, fw.tries);
                if (t >= 256 && h * 8u < t) fw.use_smem = false;
                fw.counting = false;
            }
            __syncwarp();
        }
        if constexpr (NUL) {
            if (fw.touched > 32) fw.touch_drain(static_cast<unsigned>(lane), 32);
            if (fw.touched > 0) fw.touch_drain(static_cast<unsigned>(lane), fw.touched);
        }
        if (held >= 0) {  // a wait that gave up left rows behind: release the stage all the same
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[held]);
        }
    }

    __syncthreads();
    fq = fixq<VT, WIDE>(s_emax == INT_MIN ? 0 : s_emax, hb);  // the producer warp's threads merge slots too
    ftab_flush<VT, WIDE>(sm, a, fq, &s_claims, s_null_seen != 0u);
    if (spill_on)
        for (int i = threadIdx.x; i < parts; i += blockDim.x)
            a.spill_fill[static_cast<int64_t>(i) * a.spill_ctas + blockIdx.x] = min(sfill[i], static_cast<unsigned>(a.spill_cell));
    __syncthreads();
    if (threadIdx.x == 0) publish_claims(a.counters, a.capacity, s_claims);
}

// ---------------------------------------------------------------------------------------------
// Second pass over the spill.  Work item i is partition p = i % parts, slice j = i / parts: the cells j, j + slices, ...
// of p (one per aggregation-pass CTA).  One persistent CTA per SM takes items from a counter in global memory,
// aggregates the item's rows in a bucketed shared table as large as shared memory allows and merges it into the
// global table.  The item's cells are read as one stream (a prefix of their fill counts maps a stream row to its
// cell): warp w takes the contiguous stream range [total w / W, total (w + 1) / W), finds the cell of its first row
// once and then moves its cell cursor forward step by step, so every step but the last takes 64 rows however small
// the cells are, and each warp loads its next step's records before it processes the current one.
// ---------------------------------------------------------------------------------------------
// Threads of a CTA: 1024 threads have 64 registers each, which minima, maxima and 96-bit sums do not fit (their spills go
// through the same load path as the records); 768 have 80.  Spill pass of 16.8M composite groups (SUM, COUNT, MAX of
// int64) 3.94 -> 3.36 ms, of 25M masked doubles 418 -> 293 us; a float SUM alone 566 us at 1024 and 587 us at 768.
template <int MODE>
constexpr int kFSpillThreads = (MODE & (FM_MM | FM_WIDE)) ? 768 : 1024;

template <typename VT, int MODE>
__global__ void __launch_bounds__(kFSpillThreads<MODE>, 1) gb_fspill_kernel(const AggArgs a, int32_t slices) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ unsigned long long s_claims;
    __shared__ int s_emax;
    __shared__ int s_item;
    constexpr bool VFLOAT = std::is_floating_point<VT>::value;
    constexpr bool VALS = (MODE & FM_VALS) != 0;
    constexpr bool WIDE = (MODE & FM_WIDE) != 0;
    constexpr int kWarps = kFSpillThreads<MODE> / 32;
    const FTab tab = ftab<VT>(sm, a);
    const int parts = 1 << a.spill_bits;
    const int items = parts * slices;
    unsigned* work = a.spill_fill + static_cast<int64_t>(parts) * a.spill_ctas;  // zeroed by the aggregation pass
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* pre = reinterpret_cast<int*>(sm + a.so_spill);  // pre[t]: rows of the item's cells before its t-th cell
    // First level of a two-level spill: the rows this pass's table cannot take go to the second level.
    const bool level2 = a.spill2_keys != nullptr;
    const int parts2 = level2 ? (1 << a.spill2_bits) : 0;
    unsigned* fill2 = reinterpret_cast<unsigned*>(sm + a.so_spill2);
    if (threadIdx.x == 0) s_claims = 0;
    if (level2 && blockIdx.x == 0 && threadIdx.x == 0)
        a.spill2_fill[static_cast<int64_t>(parts) * parts2] = 0u;  // the next pass's work counter
    for (;;) {
        if (threadIdx.x == 0) {
            s_item = static_cast<int>(atomicAdd(work, 1u));
            s_emax = INT_MIN;
            pre[0] = 0;
        }
        for (int i = threadIdx.x; i < parts2; i += blockDim.x) fill2[i] = 0u;
        ftab_init<VT, WIDE>(sm, a, threadIdx.x, blockDim.x);
        __syncthreads();
        const int item = s_item;
        if (item >= items) break;
        const int p = item % parts;
        const int j = item / parts;
        const int64_t cell0 = static_cast<int64_t>(p) * a.spill_ctas;
        const int ncells = (a.spill_ctas - j + slices - 1) / slices;
        for (int t = threadIdx.x; t < ncells; t += blockDim.x)
            pre[t + 1] = min(static_cast<int>(a.spill_fill[cell0 + j + slices * t]), static_cast<int>(a.spill_cell));
        __syncthreads();
        if (warp == 0) {  // inclusive scan of pre[1..ncells]: a chunk per lane, then a warp scan of the chunk sums
            const int per = (ncells + 31) / 32;
            const int t0 = 1 + lane * per;
            int sum = 0;
            for (int t = t0; t < t0 + per && t <= ncells; ++t) sum += pre[t];
            int incl = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            int run = incl - sum;
            for (int t = t0; t < t0 + per && t <= ncells; ++t) {
                run += pre[t];
                pre[t] = run;
            }
        }
        __syncthreads();
        const int total = pre[ncells];
        const int r_end = static_cast<int>(static_cast<int64_t>(total) * (warp + 1) / kWarps);
        int r0 = static_cast<int>(static_cast<int64_t>(total) * warp / kWarps);
        // The warp's cell cursor: the largest t with pre[t] <= r0 (pre[0] = 0 <= r0; empty cells share a prefix).
        int tw = 0;
        {
            int lo = 0, hi = ncells;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (pre[mid] <= r0) lo = mid;
                else hi = mid;
            }
            tw = lo;
        }
        // The step starting at stream row s0 (two rows per lane, s0 + lane and s0 + 32 + lane): moves the cursor to
        // the cell of s0, then each lane walks forward to the cell of its own rows and loads their records.
        auto load = [&](int s0, bool (&act)[2], uint64_t (&kw)[2], VT (&v)[2]) {
            while (tw + 1 < ncells && pre[tw + 1] <= s0) ++tw;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r = s0 + 32 * u + lane;
                act[u] = r < r_end;
                kw[u] = 0ull;
                v[u] = VT{};
                if (act[u]) {
                    int t = tw;
                    while (t + 1 < ncells && pre[t + 1] <= r) ++t;
                    const int64_t ri = (cell0 + j + static_cast<int64_t>(slices) * t) * a.spill_cell + (r - pre[t]);
                    if constexpr (VALS) {
                        const ulonglong2 x = reinterpret_cast<const ulonglong2*>(a.spill_keys)[ri];
                        kw[u] = x.x;
                        memcpy(&v[u], &x.y, sizeof(VT));
                    } else {
                        kw[u] = a.spill_keys[ri];
                    }
                }
            }
        };
        bool act[2], nact[2];
        uint64_t kw[2], nkw[2];
        VT v[2], nv[2];
        if (r0 < r_end) load(r0, act, kw, v);
        else act[0] = act[1] = false;
        if (VFLOAT && (MODE & FM_SUM)) {  // fixed-point scale from every warp's first rows
            int e = max(act[0] ? fexp<VT>(v[0]) : INT_MIN, act[1] ? fexp<VT>(v[1]) : INT_MIN);
            e = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0 && e != INT_MIN) atomicMax(&s_emax, e);
        }
        __syncthreads();
        const int hb = max(1, 64 - __clzll(static_cast<long long>(total)));
        const FixQ fq = fixq<VT, WIDE>(s_emax == INT_MIN ? 0 : s_emax, hb);
        FastWarp<VT, MODE> fw(a, tab, fq, &s_claims);
        fw.bshift = 32 - a.spill_bits;
        fw.fits = a.fits != 0;
        fw.probe_b = a.probe_b;
        if (level2) {
            fw.spill_ok = true;
            fw.sfill = smem_u32(fill2);
            fw.cell_cap = static_cast<unsigned>(a.spill2_cell);
            fw.part_shift = 64 - a.spill_bits - a.spill2_bits;
            fw.part_mask = static_cast<uint32_t>(parts2 - 1);
            fw.cell_base = static_cast<uint32_t>(p) * static_cast<uint32_t>(parts2);
            fw.cell_mul = 1;
            fw.spill_out = a.spill2_keys;
        }
        for (; r0 < r_end; r0 += 64) {
            const int n0 = r0 + 64;
            if (n0 < r_end) load(n0, nact, nkw, nv);
            fw.template rows<2>(act, kw, v, static_cast<unsigned>(lane));
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                act[u] = nact[u];
                kw[u] = nkw[u];
                v[u] = nv[u];
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < parts2; i += blockDim.x)
            a.spill2_fill[static_cast<int64_t>(p) * parts2 + i] = min(fill2[i], static_cast<unsigned>(a.spill2_cell));
        ftab_flush<VT, WIDE, true>(sm, a, fq, &s_claims);
        __syncthreads();
    }
    if (threadIdx.x == 0) publish_claims(a.counters, a.capacity, s_claims);
}

// Launches the fast aggregation pass: one persistent CTA per SM (exactly spill_ctas CTAs when spilling).
template <typename KT, bool COMP, typename VT, typename PT, int MODE>
int32_t launch_fast_t(const AggArgs& a, size_t smem, cudaStream_t st) {
    auto kern = gb_fast_kernel<KT, COMP, VT, PT, MODE>;
    const DeviceInfo& di = device_info();
    static std::atomic<uint64_t> allowed{0};
    const int32_t rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), allowed, "gb_fast_kernel shared memory");
    if (rc != QDB_OK) return rc;
    int64_t grid = std::min<int64_t>(di.sm_count, a.tiles);
    if (a.spill_keys) {
        if (a.spill_ctas > grid) return fail(QDB_ERROR, "gb_fast_kernel: spill plan needs more CTAs than fit");
        grid = a.spill_ctas;
    }
    if (grid < 1) return QDB_OK;
    kern<<<static_cast<unsigned>(grid), kFastThreads, smem, st>>>(a);
    note_launch();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "gb_fast_kernel launch");
    return QDB_OK;
}

template <typename VT, int MODE>
int32_t launch_fspill_t(const AggArgs& a, size_t smem, int64_t grid, int32_t slices, cudaStream_t st) {
    auto kern = gb_fspill_kernel<VT, MODE>;
    static std::atomic<uint64_t> allowed{0};
    const int32_t rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), allowed, "gb_fspill_kernel shared memory");
    if (rc != QDB_OK) return rc;
    kern<<<static_cast<unsigned>(grid), kFSpillThreads<MODE>, smem, st>>>(a, slices);
    note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "gb_fspill_kernel launch");
    return QDB_OK;
}

// Mode of a table for the fast pass: FM_VALS only when some aggregate reads the values.
inline int fast_mode(const AggArgs& a) {
    const int mm = (a.has_min || a.has_max) ? FM_MM : 0;
    const int sum = a.has_sum ? FM_SUM : 0;
    return (mm | sum) ? (FM_VALS | mm | sum) : 0;
}

// The compressed-key variant exists for single keys other than DOUBLE; plain keys run the kernel without it.  KM
// selects the fused key % m variant (instantiated in its own translation units, fast_i32_mod.cu and fast_i64_mod.cu).
template <typename KT, bool COMP, typename VT, typename PT, int MODE, bool KM>
int32_t launch_fast_z(const AggArgs& a, size_t smem, cudaStream_t st) {
    if constexpr (KM) {
        return launch_fast_t<KT, COMP, VT, PT, MODE | FM_KMOD>(a, smem, st);
    } else {
        if constexpr (!COMP && !std::is_same<KT, double>::value) {
            if (a.kz) return launch_fast_t<KT, COMP, VT, PT, MODE | FM_KZ>(a, smem, st);
        }
        if (a.kz) return fail(QDB_ERR_INVALID, "gb_fast_kernel: compressed keys need a single INT32, INT64 or FLOAT key");
        return launch_fast_t<KT, COMP, VT, PT, MODE>(a, smem, st);
    }
}

template <typename KT, bool COMP, typename VT, typename PT, bool KM>
int32_t launch_fast_m(const AggArgs& a, size_t smem, cudaStream_t st) {
    switch (fast_mode(a)) {
        case FM_VALS | FM_SUM: return launch_fast_z<KT, COMP, VT, PT, FM_VALS | FM_SUM, KM>(a, smem, st);
        case FM_VALS | FM_MM: return launch_fast_z<KT, COMP, VT, PT, FM_VALS | FM_MM, KM>(a, smem, st);
        case FM_VALS | FM_SUM | FM_MM: return launch_fast_z<KT, COMP, VT, PT, FM_VALS | FM_SUM | FM_MM, KM>(a, smem, st);
        default: return fail(QDB_ERR_INVALID, "gb_fast_kernel: unsupported aggregate set");
    }
}

// Calls with NULL masks or a row mask (single key): one instantiation per key type, value type and aggregate set.
template <typename KT, typename VT, int MODE>
int32_t launch_fast_nul_t(const AggArgs& a, size_t smem, cudaStream_t st) {
    constexpr int W = (std::is_floating_point<VT>::value && (MODE & FM_SUM)) ? FM_WIDE : 0;
    return launch_fast_t<KT, false, VT, NoPred, MODE | FM_NULL | W>(a, smem, st);
}

template <typename KT, typename VT>
int32_t launch_fast_nul_m(const AggArgs& a, size_t smem, cudaStream_t st) {
    switch (fast_mode(a)) {
        case FM_VALS | FM_SUM: return launch_fast_nul_t<KT, VT, FM_VALS | FM_SUM>(a, smem, st);
        case FM_VALS | FM_MM: return launch_fast_nul_t<KT, VT, FM_VALS | FM_MM>(a, smem, st);
        case FM_VALS | FM_SUM | FM_MM: return launch_fast_nul_t<KT, VT, FM_VALS | FM_SUM | FM_MM>(a, smem, st);
        default: return fail(QDB_ERR_INVALID, "gb_fast_kernel: unsupported aggregate set");
    }
}

template <typename KT>
int32_t launch_fast_nul_k(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st) {
    if (fast_mode(a) == 0) return launch_fast_nul_t<KT, int32_t, 0>(a, smem, st);
    switch (vk) {
        case VK_I32: return launch_fast_nul_m<KT, int32_t>(a, smem, st);
        case VK_I64: return launch_fast_nul_m<KT, int64_t>(a, smem, st);
        case VK_F32: return launch_fast_nul_m<KT, float>(a, smem, st);
        case VK_F64: return launch_fast_nul_m<KT, double>(a, smem, st);
        default: return fail(QDB_ERR_INVALID, "unsupported value type");
    }
}

template <typename KT, bool COMP, typename PT, bool KM>
int32_t launch_fast_v(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st) {
    if (fast_mode(a) == 0) return launch_fast_z<KT, COMP, int32_t, PT, 0, KM>(a, smem, st);
    switch (vk) {
        case VK_I32: return launch_fast_m<KT, COMP, int32_t, PT, KM>(a, smem, st);
        case VK_I64: return launch_fast_m<KT, COMP, int64_t, PT, KM>(a, smem, st);
        case VK_F32: return launch_fast_m<KT, COMP, float, PT, KM>(a, smem, st);
        case VK_F64: return launch_fast_m<KT, COMP, double, PT, KM>(a, smem, st);
        default: return fail(QDB_ERR_INVALID, "unsupported value type");
    }
}

template <typename KT, bool COMP, bool KM = false>
int32_t launch_fast_k(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st) {
    switch (ptype) {
        case 0: return launch_fast_v<KT, COMP, NoPred, KM>(a, vk, smem, st);
        case QDB_INT32: return launch_fast_v<KT, COMP, int32_t, KM>(a, vk, smem, st);
        case QDB_INT64: return launch_fast_v<KT, COMP, int64_t, KM>(a, vk, smem, st);
        case QDB_FLOAT: return launch_fast_v<KT, COMP, float, KM>(a, vk, smem, st);
        case QDB_DOUBLE: return launch_fast_v<KT, COMP, double, KM>(a, vk, smem, st);
        default: return fail(QDB_ERR_INVALID, "unsupported predicate column type");
    }
}

template <typename VT>
int32_t launch_fspill_m(const AggArgs& a, size_t smem, int64_t grid, int32_t slices, cudaStream_t st) {
    if constexpr (std::is_floating_point<VT>::value) {
        if (a.wide && fast_mode(a) == (FM_VALS | FM_SUM))
            return launch_fspill_t<VT, FM_VALS | FM_SUM | FM_WIDE>(a, smem, grid, slices, st);
        if (a.wide && fast_mode(a) == (FM_VALS | FM_SUM | FM_MM))
            return launch_fspill_t<VT, FM_VALS | FM_SUM | FM_MM | FM_WIDE>(a, smem, grid, slices, st);
    }
    switch (fast_mode(a)) {
        case FM_VALS | FM_SUM: return launch_fspill_t<VT, FM_VALS | FM_SUM>(a, smem, grid, slices, st);
        case FM_VALS | FM_MM: return launch_fspill_t<VT, FM_VALS | FM_MM>(a, smem, grid, slices, st);
        case FM_VALS | FM_SUM | FM_MM: return launch_fspill_t<VT, FM_VALS | FM_SUM | FM_MM>(a, smem, grid, slices, st);
        default: return fail(QDB_ERR_INVALID, "gb_fspill_kernel: unsupported aggregate set");
    }
}

// Per-key-type entry points of the fast pass, each instantiated in its key type's translation unit.
int32_t launch_fast_i32(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);
int32_t launch_fast_i64(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);
int32_t launch_fast_i32_mod(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);
int32_t launch_fast_i64_mod(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);
int32_t launch_fast_f32(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);
int32_t launch_fast_f64(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);
int32_t launch_fast_i32_nul(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st);
int32_t launch_fast_i64_nul(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st);
int32_t launch_fast_f32_nul(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st);
int32_t launch_fast_f64_nul(const AggArgs& a, ValKind vk, size_t smem, cudaStream_t st);
// The pass of tables that hold every group (groupby_few.cuh): `grid` CTAs.
int32_t launch_few_i32(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st);
int32_t launch_few_f32(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st);
int32_t launch_few_comp(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st);
int32_t launch_fast_comp(const AggArgs& a, ValKind vk, int32_t ptype, size_t smem, cudaStream_t st);

}  // namespace qdb
