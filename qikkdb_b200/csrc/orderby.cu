// ORDER BY over GROUP BY results: the permutation that sorts rows by several columns (each ascending or
// descending), and the gather that applies it with OFFSET / LIMIT.  The replacement of GPUOrderBy::OrderByColumn
// and ReOrderByIdx / ReOrderNullValuesByIdx (qikkDB/QueryEngine/GPUCore/GPUOrderBy.cuh:88-195), which the
// dispatcher runs over the result columns of a GROUP BY (a CUB radix sort per column, columns from the last to the
// first).
//
// The same order is produced here with our own stable LSD radix sort: every column, from the last to the first,
// re-sorts the current permutation by that column's key, so the first column ends up most significant and equal
// rows keep their input order.  A column's key is an order-preserving unsigned encoding of its value (integers:
// the sign bit flipped; IEEE values: all bits flipped when negative, else the sign bit set), inverted for a
// descending column; a NULL row takes the encoding of lowest(T), the value the reference writes into NULL rows
// before it sorts (TransformNullValsToSmallestVal).
//
// Two forms.  Up to kObSmallRows rows one block sorts every column in shared memory in a single launch.  More rows
// take one kernel that encodes the keys and counts all their 8-bit digits, one that scans those counts, and one
// kernel per digit (a pass whose digit is the same in every row ends at once): a tile ranks its rows, finds where its
// digits start by looking back over the counts that earlier tiles published (the chained scan of Merrill and Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016, applied to radix digits by Adinets and Merrill,
// "Onesweep", 2022), and writes its rows digit by digit from shared memory.
#include <climits>
#include <cfloat>

#include "groupby.cuh"

namespace qdb {

constexpr int kObThreads = 512;                      // 16 warps: a tile of the radix passes
constexpr int kObWarps = kObThreads / 32;
template <typename K>
constexpr int kObItems = sizeof(K) == 8 ? 8 : 12;    // rows per thread in a tile (48 KB of keys and rows to write out)
template <typename K>
constexpr int kObTile = kObThreads * kObItems<K>;
constexpr int kObSmallThreads = 1024;
constexpr int kObSmallItems = 8;                     // rows per thread of the one-block form
constexpr int kObSmallRows = kObSmallThreads * kObSmallItems;
constexpr int kObSmallCols = 8;                      // columns per launch of the one-block form

// Order-preserving unsigned encodings (ascending order of the value = ascending unsigned order).
__device__ __forceinline__ uint32_t ob_enc(int32_t v) { return static_cast<uint32_t>(v) ^ 0x80000000u; }
__device__ __forceinline__ uint64_t ob_enc(int64_t v) { return static_cast<uint64_t>(v) ^ 0x8000000000000000ull; }
__device__ __forceinline__ uint32_t ob_enc(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ uint64_t ob_enc(double v) {
    const uint64_t b = static_cast<uint64_t>(__double_as_longlong(v));
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

template <typename T>
__device__ __forceinline__ T ob_lowest() {
    if constexpr (std::is_same<T, int32_t>::value) return INT_MIN;
    else if constexpr (std::is_same<T, int64_t>::value) return LLONG_MIN;
    else if constexpr (std::is_same<T, float>::value) return -FLT_MAX;
    else return -DBL_MAX;
}

template <typename T>
__device__ __forceinline__ auto ob_key(const T* __restrict__ col, const uint64_t* __restrict__ nulls, int32_t r,
                                       bool desc) {
    T v = col[r];
    if (nulls && ((nulls[r >> 6] >> (r & 63)) & 1ull)) v = ob_lowest<T>();
    const auto k = ob_enc(v);
    return desc ? static_cast<decltype(k)>(~k) : k;
}

// Lanes of the warp with this lane's digit `d` (< 256; lanes without a row pass in == false and get 0): every lane sets
// its bit in its digit's word of the warp's 256 words, which are all zero before and after.
__device__ __forceinline__ uint32_t ob_peers(uint32_t* words, uint32_t d, bool in, int lane) {
    if (in) atomicOr(&words[d], 1u << lane);
    __syncwarp();
    const uint32_t peers = in ? words[d] : 0u;
    return peers;
}

// ---------------------------------------------------------------------------------------------
// One block, every column.  Warp w holds positions [256 w, 256 w + 256), step j the positions 32 j + lane, so rows are
// ranked in their order.  A digit that is the same in all rows is skipped.  n <= 8192 rows of 64-bit keys take 64 KB of
// keys and 32 KB of row numbers; the time is the serial chain of the passes (about 2 us each), which is still far below
// the launches of the tiled form: 1000 rows of one int32 column take one launch of 8 us instead of 13 launches, 31 us.
// ---------------------------------------------------------------------------------------------
struct ObSmallCol {
    const void* col = nullptr;
    const uint64_t* nulls = nullptr;
    int32_t type = 0;
    int32_t desc = 0;
};
struct ObSmallArgs {
    ObSmallCol c[kObSmallCols];  // in the order they are sorted by: the least significant first
    int32_t n_cols = 0;
    int32_t n = 0;
    int32_t first = 0;           // start from the identity instead of reading idx
    int32_t* idx = nullptr;
};

__global__ void __launch_bounds__(kObSmallThreads) ob_small_kernel(const ObSmallArgs a) {
    extern __shared__ __align__(16) unsigned char ob_sm[];
    const int warps = blockDim.x >> 5;
    uint64_t* keys = reinterpret_cast<uint64_t*>(ob_sm);                            // [blockDim.x * 8]
    int32_t* perm = reinterpret_cast<int32_t*>(keys + blockDim.x * kObSmallItems);    // [blockDim.x * 8]
    uint32_t* words = reinterpret_cast<uint32_t*>(perm + blockDim.x * kObSmallItems); // [warps][256] lane masks
    uint16_t* cnt = reinterpret_cast<uint16_t*>(words + warps * 256);                 // [warps][256]
    __shared__ uint32_t s_vary[2];
    __shared__ uint32_t s_dig[256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t* const w_words = words + warp * 256;
    uint16_t* const w_cnt = cnt + warp * 256;
    const int i0 = warp * (32 * kObSmallItems) + lane;
    for (int i = threadIdx.x; i < warps * 256; i += blockDim.x) words[i] = 0u;
    for (int j = 0; j < kObSmallItems; ++j) {
        const int i = i0 + 32 * j;
        if (i < a.n) perm[i] = a.first ? i : a.idx[i];  // any row numbers of the columns, not only 0..n-1
    }
    for (int c = 0; c < a.n_cols; ++c) {
        const ObSmallCol& col = a.c[c];
        const bool desc = col.desc != 0;
        if (threadIdx.x < 2) s_vary[threadIdx.x] = 0u;
        __syncthreads();
        auto key_at = [&](int r) -> uint64_t {
            switch (col.type) {
                case QDB_INT32: return ob_key(static_cast<const int32_t*>(col.col), col.nulls, r, desc);
                case QDB_INT64: return ob_key(static_cast<const int64_t*>(col.col), col.nulls, r, desc);
                case QDB_FLOAT: return ob_key(static_cast<const float*>(col.col), col.nulls, r, desc);
                default: return ob_key(static_cast<const double*>(col.col), col.nulls, r, desc);
            }
        };
        uint64_t key[kObSmallItems];
        int32_t id[kObSmallItems];
        const uint64_t k0 = key_at(perm[0]);
        uint64_t vary = 0;
#pragma unroll
        for (int j = 0; j < kObSmallItems; ++j) {
            const int i = i0 + 32 * j;
            key[j] = 0;
            id[j] = 0;
            if (i < a.n) {
                id[j] = perm[i];
                key[j] = key_at(id[j]);
                vary |= key[j] ^ k0;
            }
        }
        const uint32_t vlo = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(vary));
        const uint32_t vhi = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(vary >> 32));
        if (lane == 0) {
            atomicOr(&s_vary[0], vlo);
            atomicOr(&s_vary[1], vhi);
        }
        __syncthreads();
        vary = (static_cast<uint64_t>(s_vary[1]) << 32) | s_vary[0];
        for (int shift = 0; shift < 64; shift += 8) {
            if (((vary >> shift) & 0xffull) == 0) continue;
            for (int i = lane; i < 256; i += 32) w_cnt[i] = 0;
            __syncwarp();
            uint16_t rank[kObSmallItems];
#pragma unroll
            for (int j = 0; j < kObSmallItems; ++j) {
                const bool in = i0 + 32 * j < a.n;
                const uint32_t d = static_cast<uint32_t>(key[j] >> shift) & 0xffu;
                const uint32_t peers = ob_peers(w_words, d, in, lane);
                const uint32_t before = in ? w_cnt[d] : 0u;
                __syncwarp();
                rank[j] = static_cast<uint16_t>(before + __popc(peers & lt));
                if (in && (peers & lt) == 0u) {  // the first lane of the group
                    w_cnt[d] = static_cast<uint16_t>(before + __popc(peers));
                    w_words[d] = 0u;
                }
                __syncwarp();
            }
            __syncthreads();
            for (int d = threadIdx.x; d < 256; d += blockDim.x) {  // per digit: the warps' offsets, the digit's count
                uint32_t run = 0;
                for (int w = 0; w < warps; ++w) {
                    const uint32_t x = cnt[w * 256 + d];
                    cnt[w * 256 + d] = static_cast<uint16_t>(run);
                    run += x;
                }
                s_dig[d] = run;
            }
            __syncthreads();
            if (warp == 0) {  // exclusive scan of the 256 digit counts, eight per lane
                uint32_t v[8], sum = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    v[k] = s_dig[lane * 8 + k];
                    sum += v[k];
                }
                uint32_t incl = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                uint32_t run = incl - sum;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    s_dig[lane * 8 + k] = run;
                    run += v[k];
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kObSmallItems; ++j) {
                if (i0 + 32 * j < a.n) {
                    const uint32_t d = static_cast<uint32_t>(key[j] >> shift) & 0xffu;
                    const uint32_t p = s_dig[d] + w_cnt[d] + rank[j];
                    keys[p] = key[j];
                    perm[p] = id[j];
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kObSmallItems; ++j) {
                const int i = i0 + 32 * j;
                if (i < a.n) {
                    key[j] = keys[i];
                    id[j] = perm[i];
                }
            }
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < a.n; i += blockDim.x) a.idx[i] = perm[i];
}

// ---------------------------------------------------------------------------------------------
// The tiled form.
// ---------------------------------------------------------------------------------------------
struct ObPass {              // written by ob_meta_kernel, per digit
    uint32_t run;            // 0: every row has the same digit
    uint32_t ordinal;        // passes that run before this one
    uint32_t left;           // passes that run from this one on (1: it is the last)
    uint32_t ticket;         // next tile
};

// keys[i] = the encoding of col[idx[i]] (first: row i), idx copied beside it, and the counts of all digits.  Bound by
// the column read, a random one when a permutation is applied.
template <typename T, typename K>
__global__ void __launch_bounds__(kObThreads) ob_keys_kernel(const T* __restrict__ col,
                                                             const uint64_t* __restrict__ nulls,
                                                             const int32_t* __restrict__ idx, int64_t n, int32_t desc,
                                                             K* __restrict__ keys, int32_t* __restrict__ idx_out,
                                                             uint32_t* __restrict__ hist) {
    constexpr int D = sizeof(K);
    __shared__ uint32_t cnt[D * 256];
    for (int i = threadIdx.x; i < D * 256; i += kObThreads) cnt[i] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t step = static_cast<int64_t>(gridDim.x) * kObThreads;
    const int64_t lim = (n + 31) / 32 * 32;  // whole warps, so that votes see every lane
    for (int64_t i = blockIdx.x * static_cast<int64_t>(kObThreads) + threadIdx.x; i < lim; i += step) {
        const bool in = i < n;
        K k = 0;
        if (in) {
            const int32_t r = idx ? idx[i] : static_cast<int32_t>(i);
            k = ob_key(col, nulls, r, desc != 0);
            keys[i] = k;
            if (idx) idx_out[i] = r;
        }
        const uint32_t live = __ballot_sync(0xffffffffu, in);
        const K kf = __shfl_sync(0xffffffffu, k, 0);  // lane 0 always has a row
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const uint32_t x = static_cast<uint32_t>(k >> (8 * d)) & 0xffu;
            const uint32_t f = static_cast<uint32_t>(kf >> (8 * d)) & 0xffu;
            if (__all_sync(0xffffffffu, !in || x == f)) {  // a digit common to the warp: one add for all its rows
                if (lane == 0) atomicAdd(&cnt[d * 256 + f], __popc(live));
            } else if (in) {
                atomicAdd(&cnt[d * 256 + x], 1u);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < D * 256; i += kObThreads)
        if (cnt[i]) atomicAdd(&hist[i], cnt[i]);
}

// One block of 256 threads: hist becomes the exclusive start of every digit, and which passes run.
template <int D>
__global__ void __launch_bounds__(256) ob_meta_kernel(uint32_t* __restrict__ hist, uint32_t n, ObPass* __restrict__ pass) {
    __shared__ uint32_t ws[8];
    __shared__ uint32_t trivial[D];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < D) trivial[threadIdx.x] = 0u;
    for (int d = 0; d < D; ++d) {
        __syncthreads();
        const uint32_t c = hist[d * 256 + threadIdx.x];
        if (c == n) trivial[d] = 1u;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        uint32_t pre = 0;
        for (int w = 0; w < warp; ++w) pre += ws[w];
        hist[d * 256 + threadIdx.x] = pre + incl - c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t o = 0;
        for (int d = 0; d < D; ++d) {
            pass[d].run = trivial[d] ? 0u : 1u;
            pass[d].ordinal = o;
            pass[d].ticket = 0u;
            if (!trivial[d]) ++o;
        }
        for (int d = 0; d < D; ++d) pass[d].left = o - pass[d].ordinal;
        if (o == 0) pass[D - 1].ordinal = 0xffffffffu;  // no pass runs: the last kernel writes the identity
    }
}

__device__ __forceinline__ uint64_t ob_ld(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ob_st(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <typename K>
struct ObArgs {
    K* keys0 = nullptr;
    K* keys1 = nullptr;
    int32_t* idx = nullptr;          // row numbers, in turn with out so that the last pass writes out
    int32_t* out = nullptr;          // the permutation
    int64_t n = 0;
    int32_t first = 0;               // the permutation before the column's first pass is the identity
    const uint32_t* start = nullptr; // [digits][256]
    ObPass* pass = nullptr;
    uint64_t* state = nullptr;       // [tiles][256]
    uint32_t max_polls = 0;          // unsuccessful looks at its predecessors after which a tile helps itself
};

constexpr int64_t kObMaxPolls = 1 << 20;
constexpr int kObLook = 8;

// One pass of one tile.  state[t * 256 + d]: high word 2 p + 1 when the low word is the count of digit d in tile t, 2 p
// + 2 when it is the count in tiles 0..t (p the pass; the words of earlier passes are smaller, so the area is cleared
// once per column).  Tiles are numbered by a ticket, so a tile's predecessors are running or done; a tile that has
// polled a.max_polls times counts its predecessors' rows itself instead of waiting on.
//
// Rows leave through shared memory in digit order, so a digit's 16 rows of a tile on average (24 for 32-bit keys) go out
// in one piece.  10M rows of 64-bit keys: 98 us a digit, where histogram, scan and scatter took 117; of 32-bit keys 67 us.
// The 24 bytes read and written per row would take 36 us and the 2.2M pieces of a pass about 55 at 40 G/s; what makes up
// the rest is not settled.  Tiles of 1024 threads or 14 keys a thread, with half the pieces, tiles of 256 threads and other
// look-back widths all take 98 to 106 us, so neither the pieces nor the look-back alone bound it; the chain of the rank
// loop (an atomic, a read and a write per step and warp) and the seven barriers of a tile have not been taken apart.
template <typename K>
__global__ void __launch_bounds__(kObThreads, 2) ob_pass_kernel(const ObArgs<K> a, int p) {
    constexpr int ITEMS = kObItems<K>;
    constexpr int TILE = kObTile<K>;
    extern __shared__ __align__(16) unsigned char ob_sm[];
    K* s_keys = reinterpret_cast<K*>(ob_sm);                            // [TILE]
    int32_t* s_idx = reinterpret_cast<int32_t*>(s_keys + TILE);         // [TILE]
    uint32_t* words = reinterpret_cast<uint32_t*>(s_idx + TILE);        // [kObWarps][256] lane masks
    uint16_t* cnt = reinterpret_cast<uint16_t*>(words + kObWarps * 256);  // [kObWarps][256]
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_first[256];  // digit's first position in the tile
    __shared__ uint32_t s_glob[256];   // digit's first position in the output, less s_first
    __shared__ uint32_t s_ws[8];
    const ObPass ps = a.pass[p];
    if (!ps.run) {
        if (ps.ordinal == 0xffffffffu && a.first)  // nothing to sort: rows stay in their order
            for (int64_t i = blockIdx.x * static_cast<int64_t>(kObThreads) + threadIdx.x; i < a.n;
                 i += static_cast<int64_t>(gridDim.x) * kObThreads)
                a.out[i] = static_cast<int32_t>(i);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const int shift = 8 * p;
    const bool odd = (ps.ordinal & 1u) != 0;
    const K* __restrict__ keys_in = odd ? a.keys1 : a.keys0;
    K* __restrict__ keys_out = odd ? a.keys0 : a.keys1;
    const bool ident = a.first && ps.ordinal == 0;
    const int32_t* __restrict__ idx_in = (ps.left & 1u) ? a.idx : a.out;
    int32_t* __restrict__ idx_out = (ps.left & 1u) ? a.out : a.idx;
    if (threadIdx.x == 0) s_tile = atomicAdd(&a.pass[p].ticket, 1u);
    for (int i = threadIdx.x; i < kObWarps * 256; i += kObThreads) {
        words[i] = 0u;
        cnt[i] = 0;
    }
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t base = tile * TILE;
    const int rows = static_cast<int>(min(static_cast<int64_t>(TILE), a.n - base));
    const int i0 = warp * (32 * ITEMS) + lane;
    uint32_t* const w_words = words + warp * 256;
    uint16_t* const w_cnt = cnt + warp * 256;
    K key[ITEMS];
    int32_t id[ITEMS];
    uint16_t rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = i0 + 32 * j;
        key[j] = i < rows ? keys_in[base + i] : K(0);
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = i0 + 32 * j;
        id[j] = ident ? static_cast<int32_t>(base + i) : (i < rows ? idx_in[base + i] : 0);
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const bool in = i0 + 32 * j < rows;
        const uint32_t d = static_cast<uint32_t>(key[j] >> shift) & 0xffu;
        const uint32_t peers = ob_peers(w_words, d, in, lane);
        const uint32_t before = in ? w_cnt[d] : 0u;
        __syncwarp();
        rank[j] = static_cast<uint16_t>(before + __popc(peers & lt));
        if (in && (peers & lt) == 0u) {
            w_cnt[d] = static_cast<uint16_t>(before + __popc(peers));
            w_words[d] = 0u;
        }
        __syncwarp();
    }
    __syncthreads();
    // Digit threads: the warps' offsets, the tile's count (published at once) and, over the digits, its positions.
    uint32_t count = 0, incl = 0;
    uint64_t* const my_state = a.state + tile * 256 + threadIdx.x;
    const uint64_t f_agg = static_cast<uint64_t>(2 * p + 1) << 32, f_inc = static_cast<uint64_t>(2 * p + 2) << 32;
    if (threadIdx.x < 256) {
        for (int w = 0; w < kObWarps; ++w) {
            const uint32_t x = cnt[w * 256 + threadIdx.x];
            cnt[w * 256 + threadIdx.x] = static_cast<uint16_t>(count);
            count += x;
        }
        ob_st(my_state, (tile == 0 ? f_inc : f_agg) | count);
        incl = count;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_ws[warp] = incl;
    }
    __syncthreads();
    if (threadIdx.x < 256) {
        uint32_t pre = incl - count;
        for (int w = 0; w < warp; ++w) pre += s_ws[w];
        s_first[threadIdx.x] = pre;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (i0 + 32 * j < rows) {
            const uint32_t d = static_cast<uint32_t>(key[j] >> shift) & 0xffu;
            const uint32_t pos = s_first[d] + w_cnt[d] + rank[j];
            s_keys[pos] = key[j];
            s_idx[pos] = id[j];
        }
    }
    bool gave_up = false;
    uint32_t before = 0;
    if (threadIdx.x < 256 && tile > 0) {
        const uint64_t* st = a.state + threadIdx.x;
        uint32_t polls = 0;
        bool done = false;
        for (int64_t t = tile - 1; !done && !gave_up;) {
            // kObLook predecessors at a time, so that their loads overlap (one by one, the hundreds of tiles in flight
            // made a tile walk as many L2 round trips: 106 us a pass over 10M 64-bit keys)
            uint64_t x[kObLook];
#pragma unroll
            for (int k = 0; k < kObLook; ++k) x[k] = t - k >= 0 ? ob_ld(st + (t - k) * 256) : f_inc;
            int took = 0;
#pragma unroll
            for (int k = 0; k < kObLook; ++k) {
                if (!done && took == k && x[k] >= f_agg) {
                    before += static_cast<uint32_t>(x[k]);
                    done = x[k] >= f_inc;
                    ++took;
                }
            }
            t -= took;
            if (took == 0 && ++polls > a.max_polls) gave_up = true;
        }
        if (!gave_up) ob_st(my_state, f_inc | (before + count));
    }
    if (__syncthreads_or(gave_up ? 1 : 0)) {
        // Not expected: count the rows before this tile (words serves as the counters; its users are done).
        for (int i = threadIdx.x; i < 256; i += kObThreads) words[i] = 0u;
        __syncthreads();
        for (int64_t i = threadIdx.x; i < base; i += kObThreads)
            atomicAdd(&words[static_cast<uint32_t>(keys_in[i] >> shift) & 0xffu], 1u);
        __syncthreads();
        if (threadIdx.x < 256) {
            before = words[threadIdx.x];
            ob_st(my_state, f_inc | (before + count));
        }
    }
    if (threadIdx.x < 256) s_glob[threadIdx.x] = a.start[p * 256 + threadIdx.x] + before - s_first[threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.x; i < rows; i += kObThreads) {
        const K k = s_keys[i];
        const uint32_t g = s_glob[static_cast<uint32_t>(k >> shift) & 0xffu] + static_cast<uint32_t>(i);
        if (ps.left > 1u) keys_out[g] = k;
        idx_out[g] = s_idx[i];
    }
}

// out[i] = in[idx[offset + i]] for i < count.
template <typename T>
__global__ void ob_gather_kernel(const T* __restrict__ in, const int32_t* __restrict__ idx, int64_t offset,
                                 int64_t count, T* __restrict__ out) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[i] = in[idx[offset + i]];
}

// Null bits gathered the same way: word w of out holds the bits of rows 64 w .. 64 w + 63.
__global__ void ob_gather_nulls_kernel(const uint64_t* __restrict__ in, const int32_t* __restrict__ idx,
                                       int64_t offset, int64_t count, uint64_t* __restrict__ out) {
    for (int64_t w = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; w < (count + 63) / 64;
         w += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        uint64_t bits = 0;
        for (int b = 0; b < 64 && 64 * w + b < count; ++b) {
            const int32_t r = idx[offset + 64 * w + b];
            bits |= ((in[r >> 6] >> (r & 63)) & 1ull) << b;
        }
        out[w] = bits;
    }
}

static unsigned ob_grid(int64_t n, int threads) {
    const DeviceInfo& di = device_info();
    return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads,
                                                                        int64_t(di.sm_count) * 16)));
}

// Re-sorts the permutation `indices` (first: the identity) by one column, tiled form.
template <typename T>
static int32_t ob_column(const void* col, const uint64_t* nulls, int32_t desc, int64_t n, bool first, int32_t* indices,
                         cudaStream_t s) {
    using K = typename std::conditional<sizeof(T) == 4, uint32_t, uint64_t>::type;
    constexpr int D = sizeof(K);
    const int64_t tiles = (n + kObTile<K> - 1) / kObTile<K>;
    static std::atomic<uint64_t> allowed{0};
    int32_t rc = allow_dynamic_smem(reinterpret_cast<const void*>(ob_pass_kernel<K>), allowed, "ob_pass_kernel shared memory");
    if (rc != QDB_OK) return rc;
    // One allocation: the digit counts, the passes and the tile states (cleared), two key buffers and one of row numbers.
    const size_t hist_b = D * 256 * sizeof(uint32_t), pass_b = 256, state_b = static_cast<size_t>(tiles) * 256 * 8;
    const size_t key_b = (static_cast<size_t>(n) * sizeof(K) + 255) / 256 * 256, idx_b = (static_cast<size_t>(n) * 4 + 255) / 256 * 256;
    unsigned char* mem = nullptr;
    rc = dev_alloc(reinterpret_cast<void**>(&mem), hist_b + pass_b + state_b + 2 * key_b + idx_b, s);
    if (rc != QDB_OK) return rc;
    ObArgs<K> a;
    uint32_t* hist = reinterpret_cast<uint32_t*>(mem);
    a.start = hist;
    a.pass = reinterpret_cast<ObPass*>(mem + hist_b);
    a.state = reinterpret_cast<uint64_t*>(mem + hist_b + pass_b);
    unsigned char* q = mem + hist_b + pass_b + state_b;
    a.keys0 = reinterpret_cast<K*>(q);
    a.keys1 = reinterpret_cast<K*>(q + key_b);
    a.idx = reinterpret_cast<int32_t*>(q + 2 * key_b);
    a.out = indices;
    a.n = n;
    a.first = first ? 1 : 0;
    a.max_polls = static_cast<uint32_t>(env_int("QDB_OB_POLLS", kObMaxPolls));
    constexpr size_t smem = static_cast<size_t>(kObTile<K>) * (sizeof(K) + 4) + kObWarps * 256 * 6;
    cudaError_t e = cudaMemsetAsync(mem, 0, hist_b + pass_b + state_b, s);
    if (e == cudaSuccess) {
        const DeviceInfo& di = device_info();
        const unsigned g = static_cast<unsigned>(std::min<int64_t>((n + kObThreads - 1) / kObThreads, int64_t(di.sm_count) * 4));
        ob_keys_kernel<T, K><<<g, kObThreads, 0, s>>>(static_cast<const T*>(col), nulls, first ? nullptr : indices, n, desc,
                                                      a.keys0, a.idx, hist);
        ob_meta_kernel<D><<<1, 256, 0, s>>>(hist, static_cast<uint32_t>(n), a.pass);
        for (int p = 0; p < D; ++p) ob_pass_kernel<K><<<static_cast<unsigned>(tiles), kObThreads, smem, s>>>(a, p);
        note_launch(2 + D);
        e = cudaGetLastError();
    }
    dev_free(mem, s);
    return e == cudaSuccess ? QDB_OK : cuda_fail(e, "ORDER BY radix pass");
}

static int32_t ob_small(const ObSmallArgs& a, cudaStream_t s) {
    const int per = 32 * kObSmallItems;
    const int threads = std::max(4, (a.n + per - 1) / per) * 32;  // at least four warps share the digit scans
    const size_t smem = static_cast<size_t>(threads) * kObSmallItems * 12 + static_cast<size_t>(threads / 32) * 256 * 6;
    static std::atomic<uint64_t> allowed{0};
    const int32_t rc = allow_dynamic_smem(reinterpret_cast<const void*>(ob_small_kernel), allowed, "ob_small_kernel shared memory");
    if (rc != QDB_OK) return rc;
    ob_small_kernel<<<1, threads, smem, s>>>(a);
    note_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QDB_OK : cuda_fail(e, "ob_small_kernel");
}

static int32_t ob_check(int32_t type, const void* col, int64_t n, const int32_t* indices) {
    if (n < 0) return fail(QDB_ERR_INVALID, "qdb_order_by_column: negative row count");
    if (n > INT32_MAX) return fail(QDB_ERR_TOO_LARGE, "qdb_order_by_column: at most 2^31 - 1 rows");
    if (type != QDB_INT32 && type != QDB_INT64 && type != QDB_FLOAT && type != QDB_DOUBLE)
        return fail(QDB_ERR_INVALID, "qdb_order_by_column: column type must be INT32, INT64, FLOAT or DOUBLE");
    if (n > 0 && (!col || !indices)) return fail(QDB_ERR_INVALID, "qdb_order_by_column: null column or indices");
    return QDB_OK;
}

}  // namespace qdb

using namespace qdb;

extern "C" {

int32_t qdb_order_by_column(int32_t type, const void* col, const uint64_t* nulls, int32_t descending, int64_t n,
                            int32_t first, int32_t* indices, void* stream) {
    const int32_t rc = ob_check(type, col, n, indices);
    if (rc != QDB_OK || n == 0) return rc;
    cudaStream_t s = as_stream(stream);
    const bool f = first != 0;
    if (n <= kObSmallRows) {
        ObSmallArgs a;
        a.c[0] = ObSmallCol{col, nulls, type, descending};
        a.n_cols = 1;
        a.n = static_cast<int32_t>(n);
        a.first = f ? 1 : 0;
        a.idx = indices;
        return ob_small(a, s);
    }
    switch (type) {
        case QDB_INT32: return ob_column<int32_t>(col, nulls, descending, n, f, indices, s);
        case QDB_INT64: return ob_column<int64_t>(col, nulls, descending, n, f, indices, s);
        case QDB_FLOAT: return ob_column<float>(col, nulls, descending, n, f, indices, s);
        default: return ob_column<double>(col, nulls, descending, n, f, indices, s);
    }
}

int32_t qdb_order_by(int32_t n_cols, const int32_t* types, const void* const* cols, const uint64_t* const* nulls,
                     const int32_t* descending, int64_t n, int32_t* out_indices, void* stream) {
    if (n_cols < 1 || !types || !cols || n < 0) return fail(QDB_ERR_INVALID, "qdb_order_by: bad arguments");
    if (n > 0 && n <= kObSmallRows) {
        for (int c = n_cols - 1; c >= 0; --c) {
            const int32_t rc = ob_check(types[c], cols[c], n, out_indices);
            if (rc != QDB_OK) return rc;
        }
        for (int c = n_cols - 1; c >= 0;) {
            ObSmallArgs a;
            a.n = static_cast<int32_t>(n);
            a.first = c == n_cols - 1;
            a.idx = out_indices;
            for (; c >= 0 && a.n_cols < kObSmallCols; --c)
                a.c[a.n_cols++] = ObSmallCol{cols[c], nulls ? nulls[c] : nullptr, types[c], descending ? descending[c] : 0};
            const int32_t rc = ob_small(a, as_stream(stream));
            if (rc != QDB_OK) return rc;
        }
        return QDB_OK;
    }
    for (int c = n_cols - 1; c >= 0; --c) {
        const int32_t rc = qdb_order_by_column(types[c], cols[c], nulls ? nulls[c] : nullptr,
                                               descending ? descending[c] : 0, n, c == n_cols - 1, out_indices, stream);
        if (rc != QDB_OK) return rc;
    }
    return QDB_OK;
}

int32_t qdb_reorder(int32_t elem_bytes, const void* in, const int32_t* indices, int64_t offset, int64_t count,
                    void* out, void* stream) {
    if (count < 0 || offset < 0 || (count > 0 && (!in || !indices || !out)))
        return fail(QDB_ERR_INVALID, "qdb_reorder: bad arguments");
    if (count == 0) return QDB_OK;
    cudaStream_t s = as_stream(stream);
    const unsigned g = ob_grid(count, 256);
    switch (elem_bytes) {
        case 1: ob_gather_kernel<uint8_t><<<g, 256, 0, s>>>(static_cast<const uint8_t*>(in), indices, offset, count, static_cast<uint8_t*>(out)); break;
        case 2: ob_gather_kernel<uint16_t><<<g, 256, 0, s>>>(static_cast<const uint16_t*>(in), indices, offset, count, static_cast<uint16_t*>(out)); break;
        case 4: ob_gather_kernel<uint32_t><<<g, 256, 0, s>>>(static_cast<const uint32_t*>(in), indices, offset, count, static_cast<uint32_t*>(out)); break;
        case 8: ob_gather_kernel<uint64_t><<<g, 256, 0, s>>>(static_cast<const uint64_t*>(in), indices, offset, count, static_cast<uint64_t*>(out)); break;
        default: return fail(QDB_ERR_INVALID, "qdb_reorder: elem_bytes must be 1, 2, 4 or 8");
    }
    note_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QDB_OK : cuda_fail(e, "ob_gather_kernel");
}

int32_t qdb_reorder_nulls(const uint64_t* in, const int32_t* indices, int64_t offset, int64_t count, uint64_t* out,
                          void* stream) {
    if (count < 0 || offset < 0 || (count > 0 && (!in || !indices || !out)))
        return fail(QDB_ERR_INVALID, "qdb_reorder_nulls: bad arguments");
    if (count == 0) return QDB_OK;
    cudaStream_t s = as_stream(stream);
    ob_gather_nulls_kernel<<<ob_grid((count + 63) / 64, 256), 256, 0, s>>>(in, indices, offset, count, out);
    note_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QDB_OK : cuda_fail(e, "ob_gather_nulls_kernel");
}

}  // extern "C"
