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

// The sites with columns c0 .. c1 and rows r0 .. r1, found by the warp together
// and listed in their order; each warp looks at all sites once instead of every
// row's.  More than NEAR of them: `count` says so, and the caller looks at all.
constexpr int NEAR = 64;
__device__ __forceinline__ int sites_near(const int *sites, int n, int c0, int c1, int r0, int r1, int lane, int *list)
{
    int count = 0;
    for (int q0 = 0; q0 < n; q0 += 32) {
        const int q = q0 + lane;
        bool in = false;
        if (q < n) {
            const int c = sites[2 * q], r = sites[2 * q + 1];
            in = c >= c0 && c <= c1 && r >= r0 && r <= r1;
        }
        const unsigned m = __ballot_sync(FULL, in);
        const int at = count + __popc(m & ((1u << lane) - 1u));
        if (in && at < NEAR) list[at] = q;
        count += __popc(m);
    }
    __syncwarp();
    return count;
}

// Rows per segment (linear_pair.cu): `strips` warps side by side, `resident`
// of an SM's warps at a time.
int rows(int64_t strips, int ny, int resident, bool friction);

}  // namespace pair
}  // namespace swals
