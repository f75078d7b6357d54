// pair_common.cuh -- what the two-steps-a-pass kernels (linear_pair.cu,
// adjoint_pair.cu) share: 16-byte lanes of one-warp CTAs.
#pragma once

#include "swals_kernels.h"

namespace swals {
namespace pair {

constexpr unsigned FULL = 0xffffffffu;

template <typename R> struct Vec;
template <> struct Vec<double> { typedef double2 T; };
template <> struct Vec<float> { typedef float4 T; };

__device__ __forceinline__ void cp16(void *smem, const void *gmem, int src_bytes)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(src_bytes));
}

// A segment's share of the gauge index behind the sites: where the sites of
// `rows` rows from row `first` start.  A row without sites costs a bit test,
// however many gauges there are.  A list of the
// warp's sites, looked at from every lane on every row, had taken 17 us a step
// for 200 gauges on one row of 400^2 FP64 (now 4.8) and, past its 64 places,
// 1050 for 1000 in a block of 1200 x 800 (now 12.7).  Reading the rows' starts
// on every row instead of the bits: adjoint pairs at 3600 x 2400 FP64 63.7 us a
// step for 60.3; looking through a row's columns for its bit: 60.5.
struct GaugeRows {
    const int2 *sorted;   // column, gauge; by row, column, gauge
    int *start;           // [rows + 1]
    unsigned any;         // bit k % 32: row k may have sites

    // (smem: 4 (rows + 1) bytes; the caller synchronises, then calls ready)
    __device__ __forceinline__ GaugeRows(int *smem, const int *sites, int n, int ny, int first, int rows, int lane)
        : sorted(nullptr), start(smem), any(0u)
    {
        if (n <= 0) return;
        const int *row_start = sites + 2 * n;
        sorted = reinterpret_cast<const int2 *>(row_start + gauge_index_rows(ny));
        for (int k = lane; k <= rows; k += 32) start[k] = row_start[min(max(first + k, 0), ny)];
    }
    __device__ __forceinline__ void ready(int rows, int lane)
    {
        if (!sorted) return;
        for (int k0 = 0; k0 < rows; k0 += 32)
            any |= __ballot_sync(FULL, k0 + lane < rows && start[k0 + lane + 1] > start[k0 + lane]);
    }
    // Whether row k may have sites.
    __device__ __forceinline__ bool on(int k) const { return (any >> (k & 31)) & 1u; }

    // f(mask, hit, column - c0, gauge) for each 32 of the sites on the rows'
    // k-th row that has some in columns c0 .. c1, in order: the lanes of the
    // mask (hit) hold one.  Called by the whole warp.
    template <typename F> __device__ __forceinline__ void on_row(int k, int c0, int c1, int lane, F f) const
    {
        if (!on(k)) return;
        const int end = start[k + 1];
        int q0 = start[k];
        if (end - q0 > 64) {   // a crowded row: 32 probes find where the columns start
            const int step = (end - q0 + 31) / 32, at = q0 + lane * step;
            const unsigned before = __ballot_sync(FULL, at < end && sorted[min(at, end - 1)].x < c0);
            q0 += max(__popc(before) - 1, 0) * step;
        }
        for (; q0 < end; q0 += 32) {
            int2 s = make_int2(0x7fffffff, 0);
            if (q0 + lane < end) s = sorted[q0 + lane];
            const bool hit = s.x >= c0 && s.x <= c1;
            const unsigned m = __ballot_sync(FULL, hit);
            if (m) f(m, hit, hit ? s.x - c0 : 0, s.y);
            if (__any_sync(FULL, s.x > c1)) break;
        }
    }
};

// Rows per segment (linear_pair.cu): `strips` warps side by side, `resident`
// of an SM's warps at a time.
int rows(int64_t strips, int ny, int resident, bool friction);

}  // namespace pair
}  // namespace swals
