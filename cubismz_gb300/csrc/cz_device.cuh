// cz_device.cuh -- constants and line transforms of the block kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cz_layout.cuh"
#include "cz_line.cuh"

namespace cz {

constexpr int kBS3 = 32 * 32 * 32;
constexpr int kMaskBytes = 4096;                      // BITSETSIZE (WaveletCompressor.h:43)
constexpr int kMaxRecord = kMaskBytes + 4 * kBS3;     // BUFMAXSIZE (WaveletCompressor.h:44)
// One block's slot in the pre-LZ4 staging area: [int32 nbytes][record],
// rounded to 16 bytes and with 16 bytes of tail room for vector over-reads.
constexpr int kSlotBytes = ((4 + kMaxRecord + 15) / 16) * 16 + 16;

// Transform kinds, fixed per kernel instantiation: 1 interp, 2 lifted interp,
// 3 average-interpolating (the reference's wtype 0 and 3).
__host__ __device__ constexpr int wkind(int wtype) { return (wtype == 1 || wtype == 2) ? wtype : 3; }

template <int N, int KIND>
__device__ __forceinline__ void line_fwd(float (&v)[N])
{
    if (KIND == 3) fwd_avg<N>(v);
    else fwd_interp<N>(v, KIND == 2);
}
template <int N, int KIND>
__device__ __forceinline__ void line_inv(float (&v)[N])
{
    if (KIND == 3) inv_avg<N>(v);
    else inv_interp<N>(v, KIND == 2);
}

}  // namespace cz
