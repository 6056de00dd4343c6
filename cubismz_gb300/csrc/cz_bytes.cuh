// cz_bytes.cuh -- byte copies between shared-memory rings, inputs and outputs
// of any alignment.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cz {

// n bytes of the ring starting at ring offset r (r + n within the ring) to d
// (any alignment): 4-byte stores once d is aligned. By threads t of nt. Reads
// up to 4 bytes past r + n.
__device__ __forceinline__ void flush(uint8_t *d, const uint8_t *ring, int r, int n, int t, int nt)
{
    int h = (int)((4 - (reinterpret_cast<uintptr_t>(d) & 3)) & 3);
    if (h > n) h = n;
    if (t < h) d[t] = ring[r + t];
    const int nw = (n - h) >> 2, b = r + h, sh = 8 * (b & 3);
    const uint32_t *sw = reinterpret_cast<const uint32_t *>(ring) + (b >> 2);
    uint32_t *dw = reinterpret_cast<uint32_t *>(d + h);
    for (int i = t; i < nw; i += nt) dw[i] = sh ? __funnelshift_r(sw[i], sw[i + 1], sh) : sw[i];
    const int e = (n - h) & 3;
    if (t < e) d[h + 4 * nw + t] = ring[b + 4 * nw + t];
}

}  // namespace cz
