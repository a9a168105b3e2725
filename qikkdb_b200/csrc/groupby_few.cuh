// The aggregation pass of a table that holds every group (few groups: nothing spills), for calls over 4-byte keys (or two
// of them) and 4-byte values in which every row counts: no predicate, NULL masks, row mask or compressed keys.
//
// The staged pass (groupby_fast.cuh) keeps one CTA of 16 consumer warps per SM fed through a ring of tiles, with lists of
// passing rows, stages carried over and spill bookkeeping: 124 warp instructions per 32 rows, issued by 4.25 warps per
// scheduler at 0.59 a cycle (2^25 rows over 10 groups).  None of that is needed here, so this pass has no ring, no
// lists and no producer: kFewThreads threads per SM load their rows with 16-byte loads one step ahead and go straight
// to the table, and the shared memory the ring took holds twice as many groups.  It is bound by its instructions.
// 2^26 rows over 4 groups (int32 keys, SUM of float): 333 us staged, 199 us here; over 2000 groups, SUM/MIN/MAX/COUNT of
// int32: 430 and 327 us.  2^27 rows over 10 groups, AVG and COUNT of float: 375 us (2.9 TB/s).
//
// Other calls are faster staged.  A predicate's list leaves the table's instructions to the passing rows: 2^24 rows over
// 300 groups (int64 keys, SUM/MIN/MAX/COUNT of double) at 5 % take 100 us staged and 206 us in a form of this pass with
// predicates.  Rows of 12 and 16 bytes leave registers for two of them a thread: 2^26 rows of int64 keys and values, SUM
// over 1000 groups, 323 us staged and 531 us.
#pragma once

#include "groupby_fast.cuh"

namespace qdb {

constexpr int kFewThreads = 768;  // 24 warps, 80 registers

template <typename T, int U>
__device__ __forceinline__ void few_load(const void* col, int64_t r, int64_t n, T (&out)[U]) {
    const T* p = static_cast<const T*>(col) + r;
    static_assert(sizeof(T) == 4 && (U == 2 || U == 4), "one 8- or 16-byte load");
    if (r + U <= n) {
        if constexpr (U == 2) {
            const int2 q = __ldcs(reinterpret_cast<const int2*>(p));
            memcpy(out, &q, 8);
        } else {
            const int4 q = __ldcs(reinterpret_cast<const int4*>(p));
            memcpy(out, &q, 16);
        }
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) out[u] = r + u < n ? p[u] : T{};
    }
}

// KT, COMP, VT, MODE as gb_fast_kernel's.
template <typename KT, bool COMP, typename VT, int MODE>
__global__ void __launch_bounds__(kFewThreads, 1) gb_few_kernel(const AggArgs a) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ unsigned long long s_claims;
    __shared__ int s_emax;
    constexpr bool VFLOAT = std::is_floating_point<VT>::value;
    constexpr bool VALS = (MODE & FM_VALS) != 0;
    constexpr bool WIDE = false;
    // Rows per thread and step: four, two of composite keys (registers).
    constexpr int U = COMP ? 2 : 4;
    const int lane = threadIdx.x & 31;

    ftab_init<VT, WIDE>(sm, a, threadIdx.x, blockDim.x);
    if (threadIdx.x == 0) {
        s_claims = 0;
        s_emax = INT_MIN;
    }
    const int64_t step = static_cast<int64_t>(gridDim.x) * kFewThreads * U;
    int64_t r = (static_cast<int64_t>(blockIdx.x) * kFewThreads + threadIdx.x) * U;
    KT k0[U], k1[U];
    VT v[U];
    auto load = [&](int64_t at) {
        few_load(a.key0, at, a.n, k0);
        if constexpr (COMP) few_load(a.key1, at, a.n, k1);
        if constexpr (VALS) few_load(a.vals, at, a.n, v);
    };
    load(r);
    __syncthreads();
    // Fixed-point scale of float sums: the largest exponent of this CTA's first step of values.
    if (VFLOAT && (MODE & FM_SUM)) {
        int e = INT_MIN;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (r + u < a.n) e = max(e, fexp<VT>(v[u]));
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0 && e != INT_MIN) atomicMax(&s_emax, e);
    }
    __syncthreads();
    // Headroom of the fixed-point sums: a slot of this CTA receives fewer than 2^hb values.
    const int64_t most = (a.n + step - 1) / step * kFewThreads * U;
    const int hb = max(9, 64 - __clzll(static_cast<long long>(most)));
    const FixQ fq = fixq<VT, WIDE>(s_emax == INT_MIN ? 0 : s_emax, hb);
    const FTab tab = ftab<VT>(sm, a);
    FastWarp<VT, MODE, !COMP && sizeof(KT) == 4> fw(a, tab, fq, &s_claims);
    fw.probe_b = a.probe_b;
    int it = 0;
    for (int64_t w = r - static_cast<int64_t>(lane) * U; w < a.n; w += step, r += step) {  // w: the warp's first row
        bool act[U];
        uint64_t kw[U];
        VT cv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            act[u] = r + u < a.n;
            if constexpr (COMP) kw[u] = composite_word(static_cast<int32_t>(k0[u]), static_cast<int32_t>(k1[u]));
            else kw[u] = key_word(k0[u]);
            if constexpr (!COMP && std::is_integral<KT>::value) {
                if (a.kmod) kw[u] = key_word(kmod_key<KT>(a, k0[u]));  // GROUP BY key % m
            }
            if constexpr (VALS) cv[u] = v[u];
            else cv[u] = VT{};
        }
        if (w + step < a.n) load(r + step);
        fw.template rows_fit<U>(act, kw, cv);
        if ((++it & 255) == 0 && __any_sync(0xffffffffu, table_full(a.counters))) break;
    }
    __syncthreads();
    ftab_flush<VT, WIDE>(sm, a, fq, &s_claims);
    __syncthreads();
    if (threadIdx.x == 0) publish_claims(a.counters, a.capacity, s_claims);
}

template <typename KT, bool COMP, typename VT, int MODE>
int32_t launch_few_t(const AggArgs& a, size_t smem, int64_t grid, cudaStream_t st) {
    auto kern = gb_few_kernel<KT, COMP, VT, MODE>;
    static std::atomic<uint64_t> allowed{0};
    const int32_t rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), allowed, "gb_few_kernel shared memory");
    if (rc != QDB_OK) return rc;
    kern<<<static_cast<unsigned>(grid), kFewThreads, smem, st>>>(a);
    note_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? QDB_OK : cuda_fail(e, "gb_few_kernel launch");
}

template <typename KT, bool COMP, typename VT>
int32_t launch_few_m(const AggArgs& a, size_t smem, int64_t grid, cudaStream_t st) {
    switch (fast_mode(a)) {
        case FM_VALS | FM_SUM: return launch_few_t<KT, COMP, VT, FM_VALS | FM_SUM>(a, smem, grid, st);
        case FM_VALS | FM_MM: return launch_few_t<KT, COMP, VT, FM_VALS | FM_MM>(a, smem, grid, st);
        case FM_VALS | FM_SUM | FM_MM: return launch_few_t<KT, COMP, VT, FM_VALS | FM_SUM | FM_MM>(a, smem, grid, st);
        default: return fail(QDB_ERR_INVALID, "gb_few_kernel: unsupported aggregate set");
    }
}

template <typename KT, bool COMP>
int32_t launch_few_k(const AggArgs& a, ValKind vk, size_t smem, int64_t grid, cudaStream_t st) {
    if (fast_mode(a) == 0) return launch_few_t<KT, COMP, int32_t, 0>(a, smem, grid, st);
    switch (vk) {
        case VK_I32: return launch_few_m<KT, COMP, int32_t>(a, smem, grid, st);
        case VK_F32: return launch_few_m<KT, COMP, float>(a, smem, grid, st);
        default: return fail(QDB_ERR_INVALID, "unsupported value type");
    }
}

}  // namespace qdb
