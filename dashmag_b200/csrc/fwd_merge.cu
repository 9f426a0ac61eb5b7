// The second half of a forward whose keys were split over blocks (forward_splits, sm100.cu): each row's partial outputs,
// normalised f32, weighed by their log-sum-exp and rounded once to the queries' dtype.
//
// A warp a row, a lane D / 32 neighbouring features, so that a part is one coalesced read; the parts of a row are summed
// in their order, so the bits repeat.  Bound by launch and latency at the sizes that split (the parts of 500 queries x 32
// heads x 128 in 4 splits are 33 MB, still in L2): the blocks are brought in under the sweep's last wave.
// Side by side: 500 queries against 8200 keys, 32 / 8 heads of 128 (64 tiles, two splits) 131 -> 84 us, merge included
// (87 with a row's log-sum-exps read one after another and its features 8 bytes a lane).
#include <cuda.h>

#include "common.cuh"
#include "sm100.h"
#include "sm100_kernels.h"

namespace dash {
namespace {

constexpr int MERGE_THREADS = 256;

template <typename T, int HD>
__global__ void __launch_bounds__(MERGE_THREADS) fwd_merge_kernel(const Sm100FwdArgs a) {
    constexpr int PER = HD / 32;
    wait_before();
    const int lane = threadIdx.x & 31;
    const int64_t rows = (int64_t)a.b * a.tq * a.hq, row = (int64_t)blockIdx.x * (MERGE_THREADS / 32) + (threadIdx.x >> 5);
    if (row >= rows) return;
    // Lane s weighs part s (there are at most 32).  A part that saw no key (-inf) left nothing and is not read; every other one
    // counts, whatever its weight: a NaN, in a part's sum or in its features, is a NaN of the row, as in the unsplit sweep.
    const float part = lane < a.splits ? a.part_lse[lane * rows + row] : -INFINITY, mx = warp_max(part);
    const float weight = part != -INFINITY ? expf(part - mx) : 0.f, den = warp_sum(weight);
    const unsigned seen = __ballot_sync(0xffffffffu, part != -INFINITY);
    float num[PER];
#pragma unroll
    for (int c = 0; c < PER; ++c) num[c] = 0.f;
#pragma unroll 4
    for (int s = 0; s < a.splits; ++s) {
        const float w = __shfl_sync(0xffffffffu, weight, s);
        if (!(seen >> s & 1u)) continue;
        const float *po = a.part_o + (s * rows + row) * HD + lane * PER;
        if constexpr (PER % 4 == 0) {
#pragma unroll
            for (int c = 0; c < PER; c += 4) {
                const float4 x = *reinterpret_cast<const float4 *>(po + c);
                num[c] = fmaf(w, x.x, num[c]);
                num[c + 1] = fmaf(w, x.y, num[c + 1]);
                num[c + 2] = fmaf(w, x.z, num[c + 2]);
                num[c + 3] = fmaf(w, x.w, num[c + 3]);
            }
        } else {
            const float2 x = *reinterpret_cast<const float2 *>(po);
            num[0] = fmaf(w, x.x, num[0]);
            num[1] = fmaf(w, x.y, num[1]);
        }
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
    struct alignas(2 * PER) Out { T e[PER]; } out;   // a lane's features in one store
#pragma unroll
    for (int c = 0; c < PER; ++c) out.e[c] = Num<T>::from_f32(num[c] * inv);
    *reinterpret_cast<Out *>(static_cast<T *>(a.out) + row * HD + lane * PER) = out;
    if (lane == 0) a.lse[row] = den > 0.f ? (float)((double)mx + log((double)den)) : -INFINITY;
}

template <typename T>
cudaError_t merge_t(const Sm100FwdArgs &a, cudaStream_t stream) {
    const int64_t rows = (int64_t)a.b * a.tq * a.hq;
    const dim3 grid((unsigned)((rows + MERGE_THREADS / 32 - 1) / (MERGE_THREADS / 32)));
    return launch_beside(a.d == 64 ? fwd_merge_kernel<T, 64> : a.d == 128 ? fwd_merge_kernel<T, 128> : fwd_merge_kernel<T, 256>, grid,
                         MERGE_THREADS, 0, stream, true, a);
}

}  // namespace

cudaError_t launch_fwd_merge(int dtype, const Sm100FwdArgs &a, cudaStream_t stream) {
    return dtype == DASH_ATTN_BF16 ? merge_t<__nv_bfloat16>(a, stream) : merge_t<__half>(a, stream);
}

}  // namespace dash
