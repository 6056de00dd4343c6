// cz_refit.cu -- the inverse transform as a linear operator W, its adjoint
// W^T, and the least-squares refit of the retained coefficients.
//
// Interpolating wavelets are not orthogonal, so keeping the thresholded
// forward coefficients does not minimise the reconstruction error. With the
// significance mask M fixed by the plain path, the refit solves
//   min_c || x - W (M c) ||^2
// per block by CGLS (conjugate gradients on the normal equations, written on
// the residual), starting from the plain survivors. The record then carries
// the refit survivors under the same mask, so the stream layout, the chunking
// and the decoder are unchanged.
//
// W is the reference's iwt (FullWaveletTransform.h:51-56, sweep order of
// WaveletsOnInterval.h:249-276) evaluated in binary32 with its stencils as
// plain linear maps; W^T applies the transposed 1D operators in the reverse
// order. Both work on the kernels' block layout (cz_layout.cuh); the C-ABI
// entry points take and return coefficients in the reference's positional
// layout, the layout FullTransformEngine::fwt leaves in place.
#include "cz_block.cuh"
#include "cz_layout.cuh"

namespace cz {

// ------------------------------------------------------------ 1D operators
// Stencil coefficients are read into constexpr locals so that they fold
// into immediates (the coefficient tables are host-side constexpr arrays).
template <class S>
__device__ __forceinline__ float dot4(float a, float b, float c, float d)
{
    constexpr float k0 = S::c[0], k1 = S::c[1], k2 = S::c[2], k3 = S::c[3];
    return __fmaf_rn(k3, d, __fmaf_rn(k2, c, __fmaf_rn(k1, b, k0 * a)));
}
template <class S>
__device__ __forceinline__ float dot3(float a, float b, float c)
{
    constexpr float k0 = S::c[0], k1 = S::c[1], k2 = S::c[2];
    return __fmaf_rn(k2, c, __fmaf_rn(k1, b, k0 * a));
}
template <class S>
__device__ __forceinline__ void axpy4(float (&s)[16], int i, float g)  // s[i..i+3] += c * g
{
    constexpr float k0 = S::c[0], k1 = S::c[1], k2 = S::c[2], k3 = S::c[3];
    s[i] = __fmaf_rn(k0, g, s[i]);
    s[i + 1] = __fmaf_rn(k1, g, s[i + 1]);
    s[i + 2] = __fmaf_rn(k2, g, s[i + 2]);
    s[i + 3] = __fmaf_rn(k3, g, s[i + 3]);
}
template <class S>
__device__ __forceinline__ void axpy3(float (&s)[16], int i, float g)
{
    constexpr float k0 = S::c[0], k1 = S::c[1], k2 = S::c[2];
    s[i] = __fmaf_rn(k0, g, s[i]);
    s[i + 1] = __fmaf_rn(k1, g, s[i + 1]);
    s[i + 2] = __fmaf_rn(k2, g, s[i + 2]);
}

// Inverse line transform (WaveletsOnInterval.h:131-152, :181-198) as a
// linear map: [s | d] -> samples.
template <int N, int KIND>
__device__ __forceinline__ void lin_inv(float (&v)[N])
{
    constexpr int H = N / 2;
    float s[H], d[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        d[i] = v[H + i];
        s[i] = KIND == 2 ? __fmaf_rn(-0.5f, d[i], v[i]) : v[i];
    }
    if (KIND != 3) {
        float o[H];
        o[0] = dot4<W1F>(s[0], s[1], s[2], s[3]);
#pragma unroll
        for (int i = 1; i < H - 2; ++i) o[i] = dot4<W1M>(s[i - 1], s[i], s[i + 1], s[i + 2]);
        o[H - 2] = dot4<W1O>(s[H - 4], s[H - 3], s[H - 2], s[H - 1]);
        o[H - 1] = dot4<W1L>(s[H - 4], s[H - 3], s[H - 2], s[H - 1]);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            v[2 * i] = s[i];
            v[2 * i + 1] = o[i] + d[i];
        }
    } else {
        v[0] = dot3<P0F>(s[0], s[1], s[2]) - d[0];
        v[1] = dot3<P1F>(s[0], s[1], s[2]) + d[0];
#pragma unroll
        for (int i = 1; i < H - 1; ++i) {
            v[2 * i] = dot3<P0M>(s[i - 1], s[i], s[i + 1]) - d[i];
            v[2 * i + 1] = dot3<P1M>(s[i - 1], s[i], s[i + 1]) + d[i];
        }
        v[N - 2] = dot3<P0L>(s[H - 3], s[H - 2], s[H - 1]) - d[H - 1];
        v[N - 1] = dot3<P1L>(s[H - 3], s[H - 2], s[H - 1]) + d[H - 1];
    }
}

// Its transpose: samples -> [s | d].
template <int N, int KIND>
__device__ __forceinline__ void lin_inv_t(float (&v)[N])
{
    constexpr int H = N / 2;
    float s[16], d[H];
    if (KIND != 3) {
#pragma unroll
        for (int i = 0; i < H; ++i) {
            s[i] = v[2 * i];
            d[i] = v[2 * i + 1];
        }
        axpy4<W1F>(s, 0, d[0]);
#pragma unroll
        for (int i = 1; i < H - 2; ++i) axpy4<W1M>(s, i - 1, d[i]);
        axpy4<W1O>(s, H - 4, d[H - 2]);
        axpy4<W1L>(s, H - 4, d[H - 1]);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            v[i] = s[i];
            v[H + i] = KIND == 2 ? __fmaf_rn(-0.5f, s[i], d[i]) : d[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < H; ++i) {
            s[i] = 0.f;
            d[i] = v[2 * i + 1] - v[2 * i];
        }
        axpy3<P0F>(s, 0, v[0]);
        axpy3<P1F>(s, 0, v[1]);
#pragma unroll
        for (int i = 1; i < H - 1; ++i) {
            axpy3<P0M>(s, i - 1, v[2 * i]);
            axpy3<P1M>(s, i - 1, v[2 * i + 1]);
        }
        axpy3<P0L>(s, H - 3, v[N - 2]);
        axpy3<P1L>(s, H - 3, v[N - 1]);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            v[i] = s[i];
            v[H + i] = d[i];
        }
    }
}

// ------------------------------------------------------------ 3D operators
// W's sweeps: level 8 x, z, y; level 16 y, x, z; level 32 z, y, x (the decode
// kernel's order); W^T runs the transposed sweeps backwards. What bounds them
// is shared memory (every sweep moves the block in and out) and the barriers
// between sweeps, so sweeps that share lines or planes are one pass:
//   * a warp owns two x-y planes (z = warp, warp + 16) and does y and x of
//     level 32 there, ordered by __syncwarp; the x lines stay in registers
//     for what follows;
//   * a thread owns two z lines (x = lane, y = warp, warp + 16); in the
//     corner z of level 16 and of level 32 are one pass over the line;
//   * y of level 8 and of level 16 are one pass over a line; the 16^3
//     corner's y and x stay in a warp's plane; one warp does x and z of
//     level 8 while the others take the z lines outside the corner.
// Four barriers instead of nine. W and W^T of 512 blocks: 147 -> 77 us
// together (40 us at the memory's rate).
template <int N, int KIND, bool T>
__device__ __forceinline__ void lin_head(float (&v)[2 * N])  // the first N entries of a line
{
    float t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = v[i];
    if (T) lin_inv_t<N, KIND>(t);
    else lin_inv<N, KIND>(t);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = t[i];
}

// Keep bits of the coefficients that a thread's lines end with (all set where a
// line's head goes on to a further pass): z lines of level 32, the y line of
// level 16, x lines of level 8.
struct Keep {
    unsigned z[2], y, x[2];
};
template <int N>
__device__ __forceinline__ void keep_only(float (&v)[N], unsigned m)
{
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = (m >> i) & 1u ? v[i] : 0.f;
}

// Two passes of level 8 by one warp: x then z, or (T) z then x.
template <int KIND, bool T, bool MASK = false>
__device__ __forceinline__ void corner8(float *sb, const Keep &kp = Keep())
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const bool xline = (pass == 0) != T;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int a = lane & 7, c = (lane >> 3) + 4 * h;
            float v[8];
            if (xline) {
                ld_line<8, 0>(sb, pidx(0, a, c), v);
                if (T) lin_inv_t<8, KIND>(v);
                else lin_inv<8, KIND>(v);
                if (MASK) keep_only<8>(v, kp.x[h]);
                st_line<8, 0>(sb, pidx(0, a, c), v);
            } else {
                ld_line<8, 2>(sb, pidx(a, c, 0), v);
                if (T) lin_inv_t<8, KIND>(v);
                else lin_inv<8, KIND>(v);
                st_line<8, 2>(sb, pidx(a, c, 0), v);
            }
        }
        __syncwarp();
    }
}

// Level 8's y, level 16's y and x in plane z = warp of the 16^3 corner (T:
// x and y of level 16, y of level 8). Every warp.
template <int KIND, bool T, bool MASK = false>
__device__ __forceinline__ void corner16(float *sb, const Keep &kp = Keep())
{
    const int lane = threadIdx.x & 31, z = threadIdx.x >> 5;
    float v[16];
    if (T && lane < 16) {
        ld_line<16, 0>(sb, pidx(0, lane, z), v);
        lin_inv_t<16, KIND>(v);
        st_line<16, 0>(sb, pidx(0, lane, z), v);
    }
    __syncwarp();
    if (lane < 16) {
        ld_line<16, 1>(sb, pidx(lane, 0, z), v);
        if (!T && lane < 8 && z < 8) lin_head<8, KIND, T>(v);
        if (T) lin_inv_t<16, KIND>(v);
        else lin_inv<16, KIND>(v);
        if (T && lane < 8 && z < 8) lin_head<8, KIND, T>(v);
        if (MASK) keep_only<16>(v, kp.y);
        st_line<16, 1>(sb, pidx(lane, 0, z), v);
    }
    __syncwarp();
    if (!T && lane < 16) {
        ld_line<16, 0>(sb, pidx(0, lane, z), v);
        lin_inv<16, KIND>(v);
        st_line<16, 0>(sb, pidx(0, lane, z), v);
    }
}

// The warp's plane z at level 32: y, then x; lane y's x line is left in v.
template <int KIND>
__device__ __forceinline__ void plane_inv(float *sb, int z, float (&v)[32])
{
    const int lane = threadIdx.x & 31;
    ld_line<32, 1>(sb, pidx(lane, 0, z), v);
    lin_inv<32, KIND>(v);
    st_line<32, 1>(sb, pidx(lane, 0, z), v);
    __syncwarp();
    ld_line<32, 0>(sb, pidx(0, lane, z), v);
    lin_inv<32, KIND>(v);
}
// Its transpose: lane y's x line in v; x, then y, stored.
template <int KIND>
__device__ __forceinline__ void plane_adj(float *sb, int z, float (&v)[32])
{
    const int lane = threadIdx.x & 31;
    lin_inv_t<32, KIND>(v);
    st_line<32, 0>(sb, pidx(0, lane, z), v);
    __syncwarp();
    ld_line<32, 1>(sb, pidx(lane, 0, z), v);
    lin_inv_t<32, KIND>(v);
    st_line<32, 1>(sb, pidx(lane, 0, z), v);
}

// z passes of W^T and its corner, from synchronised planes to a synchronised
// block (MASK: M W^T).
template <int KIND, bool MASK = false>
__device__ __forceinline__ void z_adj(float *sb, const Keep &kp = Keep())
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[32];
    {
        const int base = pidx(lane, warp, 0);
        ld_line<32, 2>(sb, base, v);
        lin_inv_t<32, KIND>(v);
        if (lane < 16) lin_head<16, KIND, true>(v);
        if (MASK) keep_only<32>(v, kp.z[0]);
        st_line<32, 2>(sb, base, v);
    }
    __syncthreads();
    corner16<KIND, true, MASK>(sb, kp);
    __syncthreads();
    if (warp == 0) corner8<KIND, true, MASK>(sb, kp);
    {
        const int base = pidx(lane, warp + 16, 0);
        ld_line<32, 2>(sb, base, v);
        lin_inv_t<32, KIND>(v);
        if (MASK) keep_only<32>(v, kp.z[1]);
        st_line<32, 2>(sb, base, v);
    }
    __syncthreads();
}

// Dense element i of a block (x fastest) and its padded shared address.
__device__ __forceinline__ int pad_of(int i) { return pidx(i & 31, (i >> 5) & 31, i >> 10); }

// ------------------------------------------------------------ dense kernels
// Row (py, pz) of a block in the reference's positional layout, entry px:
// its place in the kernels' layout (cz_layout.cuh). 32 consecutive px of a row
// outside the corner are a z line: coalesced in global memory, and SZ = 1
// mod 32 spreads them over the banks.
__device__ __forceinline__ int pad_of_row(int px, int py, int pz)
{
    if (px >= 16 || py >= 16 || pz >= 16) return pidx(py, pz, px);
    if (px >= 8 || py >= 8 || pz >= 8) return pidx(pz, px, py);
    return pidx(px, py, pz);
}

template <int KIND>
__global__ void __launch_bounds__(kNT, 1) iwt_linear_kernel(const float *coef, float *out, long long nblocks)
{
    extern __shared__ __align__(16) unsigned char smem[];
    float *sb = reinterpret_cast<float *>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long g = blockIdx.x; g < nblocks; g += gridDim.x) {
        const float *src = coef + g * kBS3 + lane;
        float v[32];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int pz = warp + 16 * h;
#pragma unroll
            for (int py = 0; py < 32; ++py) v[py] = __ldcs(src + 32 * (py + 32 * pz));
#pragma unroll
            for (int py = 0; py < 32; ++py) sb[pad_of_row(lane, py, pz)] = v[py];
        }
        __syncthreads();
        // the next block on its way to L2 meanwhile: two lines per thread
        if (g + gridDim.x < nblocks) {
            const float *nx = coef + (g + gridDim.x) * kBS3;
            for (int i = threadIdx.x; i < kBS3 / 32; i += kNT) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + 32 * i));
        }
        if (warp == 0) corner8<KIND, false>(sb);
        {
            const int base = pidx(lane, warp + 16, 0);
            ld_line<32, 2>(sb, base, v);
            lin_inv<32, KIND>(v);
            st_line<32, 2>(sb, base, v);
        }
        __syncthreads();
        corner16<KIND, false>(sb);
        __syncthreads();
        {
            const int base = pidx(lane, warp, 0);
            ld_line<32, 2>(sb, base, v);
            if (lane < 16) lin_head<16, KIND, false>(v);
            lin_inv<32, KIND>(v);
            st_line<32, 2>(sb, base, v);
        }
        __syncthreads();
        float *dst = out + g * kBS3 + lane;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int z = warp + 16 * h;
            plane_inv<KIND>(sb, z, v);
            st_line<32, 0>(sb, pidx(0, lane, z), v);
            __syncwarp();
#pragma unroll
            for (int y = 0; y < 32; ++y) __stcs(dst + 32 * (y + 32 * z), sb[pidx(lane, y, z)]);
        }
        __syncthreads();
    }
}

template <int KIND>
__global__ void __launch_bounds__(kNT, 1) iwt_adjoint_kernel(const float *in, float *coef, long long nblocks)
{
    extern __shared__ __align__(16) unsigned char smem[];
    float *sb = reinterpret_cast<float *>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long g = blockIdx.x; g < nblocks; g += gridDim.x) {
        const float *src = in + g * kBS3 + lane;
        float v[32];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int z = warp + 16 * h;
#pragma unroll
            for (int y = 0; y < 32; ++y) v[y] = __ldcs(src + 32 * (y + 32 * z));
#pragma unroll
            for (int y = 0; y < 32; ++y) sb[pidx(lane, y, z)] = v[y];
            __syncwarp();
            ld_line<32, 0>(sb, pidx(0, lane, z), v);
            __syncwarp();
            plane_adj<KIND>(sb, z, v);
        }
        __syncthreads();
        if (g + gridDim.x < nblocks) {
            const float *nx = in + (g + gridDim.x) * kBS3;
            for (int i = threadIdx.x; i < kBS3 / 32; i += kNT) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + 32 * i));
        }
        z_adj<KIND>(sb);
        float *dst = coef + g * kBS3 + lane;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int pz = warp + 16 * h;
#pragma unroll
            for (int py = 0; py < 32; ++py) __stcs(dst + 32 * (py + 32 * pz), sb[pad_of_row(lane, py, pz)]);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ refit
// Sum of the threads' v >= 0 in binary64: lanes by a shuffle tree, then the
// warps' sums one after the other. Binary64 runs at 2 lanes a cycle and SM, so
// this took 10 k cycles when every thread added 16 sums and divided, 3.5 k
// with the last part in one warp. A sum that binary64 holds exactly does not
// depend on the order: where the exponents span 20 bits at most (24 + 20 + 9
// bits for 512 values make 53), it is formed in integers; else as described.
// then(sum) runs in warp 0, before the closing barrier.
struct SumPart {
    double d;              // a warp's sum
    unsigned long long s;  // the same in units of 2^(lo - 150), if exact
    int lo, hi;            // exponent fields of its smallest and largest entry; hi 255: not exact
};
constexpr int kSumSpan = 20, kNoExp = 1 << 14;

// sum of x < 2^54 / lanes over the warp
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long x)
{
    const unsigned l = __reduce_add_sync(0xffffffffu, (unsigned)x & 0x7ffffffu);
    const unsigned h = __reduce_add_sync(0xffffffffu, (unsigned)(x >> 27));
    return ((unsigned long long)h << 27) + l;
}
// x units of 2^(lo - 150), x < 2^53 + 1
__device__ __forceinline__ double from_units(unsigned long long x, int lo)
{
    return x ? __longlong_as_double(__double_as_longlong((double)x) + ((long long)(lo - 150) << 52)) : 0.0;
}

template <class F>
__device__ __forceinline__ void block_sum(float v, SumPart *part, F &&then)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const unsigned b = __float_as_uint(v);
        const int e = (int)(b >> 23);  // from 256 on: a NaN's sign
        const int lo = __reduce_min_sync(0xffffffffu, b ? e : kNoExp);
        const int hi = __reduce_max_sync(0xffffffffu, b ? e : 0);
        const bool exact = lo > 0 && hi < 255 && hi - lo <= kSumSpan;  // also without entries: lo > hi
        SumPart p;
        p.lo = lo;
        p.hi = exact ? hi : 255;
        p.s = 0;
        if (exact) {
            p.s = warp_sum(b ? (unsigned long long)((b & 0x7fffffu) | 0x800000u) << (e - lo) : 0ull);
        } else {
            double t = v;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            p.d = t;
        }
        if (lane == 0) {
            if (exact) p.d = from_units(p.s, lo);
            part[warp] = p;
        }
    }
    __syncthreads();
    if (warp == 0) {
        const SumPart p = part[lane & (kNW - 1)];
        const int lo = __reduce_min_sync(0xffffffffu, p.lo), hi = __reduce_max_sync(0xffffffffu, p.hi);
        double t = 0;
        if (hi < 255 && hi - lo <= kSumSpan) {
            t = from_units(warp_sum(lane < kNW && p.s ? p.s << (p.lo - lo) : 0ull), lo);
        } else {
#pragma unroll 1
            for (int w = 0; w < kNW; ++w) t += part[w].d;
        }
        then(t);
    }
    __syncthreads();
}

// Per block: the forward transform and thresholding of the encode kernel,
// CGLS on min ||x - W M c||^2 from the plain survivors, then the record.
//
// A step is bound by shared memory and by the latency between barriers (one
// block fills an SM's shared memory, so there is nothing else to run). The
// iterates c, p (coefficients) and r (residual), 128 KB each, are laid out by
// the thread that uses them, [float4 k of the line][thread]: coalesced, and
// nobody else reads them. c, p and the rest of r live in L2 (`scratch`),
// kRShared of r's 16 parts in the shared memory that record emission needs
// later (2.30 -> 2.24 ms).
//   * c and p go along the thread's two z lines: c += alpha p (of the step
//     before) and p = s + beta p happen where W's z pass loads the lines;
//   * r goes along the thread's two x lines: q = W p is left in registers by
//     W's x pass, ||q||^2 comes from there, r -= alpha q and W^T's x pass follow
//     in the same registers;
//   * M is applied by W^T's last store of each line.
// So the block passes through shared memory 11 times a step instead of 22,
// with 11 barriers instead of 25. 512 blocks, 30 steps: 3.64 -> 2.24 ms.
// Holding p in registers from one step to the next, or loading it ahead of the
// sums, spilled or gained nothing (2.32 ms, 2.51 ms).
constexpr int kRShared = 10;  // 80 KB beside the block and the masks
constexpr int kRefitSmem = kSmOff + kRShared * kNT * 16 > kSmBytes ? kSmOff + kRShared * kNT * 16 : kSmBytes;
template <int KIND>
__global__ void __launch_bounds__(kNT, 1)
refit_kernel(const CzField *fields, int nfields, long long total_blocks, int zerobits, int shuffle, int iters,
             uint8_t *stage, int *rec_bytes, unsigned long long *queue, float *scratch, CzChunks chunks)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const Shared s = carve(smem);
    __shared__ long long s_ticket;
    __shared__ SumPart part[kNW];
    __shared__ double s_gamma;
    __shared__ float s_ratio;
    __shared__ int s_go;
    const uint32_t zmask = zerobits > 0 ? ~((1u << zerobits) - 1u) : 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4 *Cv = reinterpret_cast<float4 *>(scratch + (size_t)blockIdx.x * 3 * kBS3) + tid, *Pv = Cv + kBS3 / 4,
           *Rv = Pv + kBS3 / 4;
    float4 *Rs = reinterpret_cast<float4 *>(smem + kSmOff) + tid;
    float *sb = s.sb;

    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_ticket = (long long)atomicAdd(queue, 1ull);
        __syncthreads();
        const long long g = s_ticket;
        if (g >= total_blocks) break;
        const BlockRef ref = locate(fields, nfields, g);
        const float eps = ref.f->eps;
        // ---- forward transform and masks (the encode kernel's sequence)
        for (int l = threadIdx.x; l < 1024; l += kNT) {
            const int y = l & 31, z = l >> 5;
            const float4 *row = reinterpret_cast<const float4 *>(ref.f->data + row_offset(ref, y, z));
            float v[32];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float4 q = __ldg(row + k);
                v[4 * k] = q.x;
                v[4 * k + 1] = q.y;
                v[4 * k + 2] = q.z;
                v[4 * k + 3] = q.w;
            }
            line_fwd<32, KIND>(v);
            st_line<32, 0>(sb, pidx(0, y, z), v);
        }
        __syncthreads();
        sweep_fwd<32, 1, KIND>(sb);
        __syncthreads();
        for (int l = threadIdx.x; l < 1024; l += kNT) {
            const int x = l & 31, y = l >> 5;
            const int base = pidx(x, y, 0);
            float v[32];
            ld_line<32, 2>(sb, base, v);
            line_fwd<32, KIND>(v);
            st_line<32, 2>(sb, base, v);
            emit32(s, x, y, keep_bits<32>(v, eps));
        }
        __syncthreads();
        sweep_fwd<16, 2, KIND>(sb);
        __syncthreads();
        sweep_fwd<16, 0, KIND>(sb);
        __syncthreads();
        if (threadIdx.x < 256) {
            const int x = threadIdx.x & 15, z = threadIdx.x >> 4;
            const int base = pidx(x, 0, z);
            float v[16];
            ld_line<16, 1>(sb, base, v);
            line_fwd<16, KIND>(v);
            st_line<16, 1>(sb, base, v);
            emit16(s, x, z, keep_bits<16>(v, eps));
        }
        __syncthreads();
        sweep_fwd<8, 1, KIND>(sb);
        __syncthreads();
        sweep_fwd<8, 2, KIND>(sb);
        __syncthreads();
        if (threadIdx.x < 64) {
            const int y = threadIdx.x & 7, z = threadIdx.x >> 3;
            const int base = pidx(0, y, z);
            float v[8];
            ld_line<8, 0>(sb, base, v);
            line_fwd<8, KIND>(v);
            st_line<8, 0>(sb, base, v);
            emit8(s, y, z, keep_bits<8>(v, eps));
        }
        __syncthreads();
        // The keep bits in kernel layout (word y + 32 z, bit x), built once
        // per block by warp votes into the emission stage, which is idle
        // until the record is written; then those of the thread's z lines.
        uint32_t *km = reinterpret_cast<uint32_t *>(s.stage);
        for (int row = warp; row < 1024; row += kNW) {
            const int m = mask_index(lane, row & 31, row >> 5);
            const unsigned w = __ballot_sync(0xffffffffu, (s.mask32[m >> 5] >> (m & 31)) & 1u);
            if (lane == 0) km[row] = w;
        }
        __syncthreads();
        Keep kp = {{0, 0}, 0, {0, 0}};
#pragma unroll 8
        for (int z = 0; z < 32; ++z) {
            kp.z[0] |= (km[warp + 32 * z] >> lane & 1u) << z;
            kp.z[1] |= (km[warp + 16 + 32 * z] >> lane & 1u) << z;
        }
#pragma unroll 8
        for (int y = 0; y < 16; ++y) kp.y |= (km[y + 32 * warp] >> lane & 1u) << y;
        kp.x[0] = km[(lane & 7) + 32 * (lane >> 3)];
        kp.x[1] = km[(lane & 7) + 32 * (4 + (lane >> 3))];
        const unsigned zm[2] = {kp.z[0], kp.z[1]};
        if (lane < 16) kp.z[0] |= 0xffffu;
        if (lane < 8 && warp < 8) kp.y |= 0xffu;
        // Entries 4 k .. 4 k + 3 of the thread's z line h, from the block to the
        // iterate that W is applied to.
        enum { kStart, kFirst, kStep };  // c0 = M c; p = s; c += alpha p, p = s + beta p
        float alpha = 0.f, beta = 0.f;
        int mode = kStart;
        bool pending = false;  // c += alpha p of the last step is still to come
        auto load4 = [&](float (&v)[32], int h, int k) {
            const unsigned m = mode == kStart ? zm[h] >> (4 * k) : 15u;
            float4 t;
            t.x = (m & 1u) ? v[4 * k] : 0.f;
            t.y = (m & 2u) ? v[4 * k + 1] : 0.f;
            t.z = (m & 4u) ? v[4 * k + 2] : 0.f;
            t.w = (m & 8u) ? v[4 * k + 3] : 0.f;
            const int at = (8 * h + k) * kNT;
            if (mode == kStart) {
                Cv[at] = t;
            } else {
                if (mode == kStep) {
                    const float4 p = Pv[at];
                    float4 c = Cv[at];
                    c.x = __fmaf_rn(alpha, p.x, c.x);
                    c.y = __fmaf_rn(alpha, p.y, c.y);
                    c.z = __fmaf_rn(alpha, p.z, c.z);
                    c.w = __fmaf_rn(alpha, p.w, c.w);
                    Cv[at] = c;
                    t.x = __fmaf_rn(beta, p.x, t.x);
                    t.y = __fmaf_rn(beta, p.y, t.y);
                    t.z = __fmaf_rn(beta, p.z, t.z);
                    t.w = __fmaf_rn(beta, p.w, t.w);
                }
                Pv[at] = t;
            }
            v[4 * k] = t.x;
            v[4 * k + 1] = t.y;
            v[4 * k + 2] = t.z;
            v[4 * k + 3] = t.w;
        };

        for (int it = -1;; ++it) {  // -1: the residual of c0
            // ---- q = W c0 or W p; lane y's x lines of the warp's planes in q
            float v[32];
            if (lane < 16) {  // the corner first: levels 8 and 16 need it whole
                const int base = pidx(lane, warp, 0);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = sb[base + j * SZ];
#pragma unroll
                for (int k = 0; k < 4; ++k) load4(v, 0, k);
#pragma unroll
                for (int j = 0; j < 16; ++j) sb[base + j * SZ] = v[j];
            }
            __syncthreads();
            if (warp == 0) corner8<KIND, false>(sb);
            {
                const int base = pidx(lane, warp + 16, 0);
                ld_line<32, 2>(sb, base, v);
#pragma unroll
                for (int k = 0; k < 8; ++k) load4(v, 1, k);
                lin_inv<32, KIND>(v);
                st_line<32, 2>(sb, base, v);
            }
            __syncthreads();
            corner16<KIND, false>(sb);
            __syncthreads();
            {
                const int base = pidx(lane, warp, 0);
                ld_line<32, 2>(sb, base, v);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k >= 4 || lane >= 16) load4(v, 0, k);
                if (lane < 16) lin_head<16, KIND, false>(v);
                lin_inv<32, KIND>(v);
                st_line<32, 2>(sb, base, v);
            }
            __syncthreads();
            float q[2][32];
            float acc = 0.f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                plane_inv<KIND>(sb, warp + 16 * h, q[h]);
#pragma unroll
                for (int j = 0; j < 32; ++j) acc = __fmaf_rn(q[h][j], q[h][j], acc);
            }
            // ---- alpha = gamma / ||q||^2
            if (it >= 0) {
                block_sum(acc, part, [&](double delta) {
                    if (lane == 0) {
                        s_go = delta > 0.0;
                        s_ratio = delta > 0.0 ? (float)(s_gamma / delta) : 0.f;
                    }
                });
                alpha = s_ratio;
                pending = s_go != 0;
                if (!pending) break;  // nothing left to gain: c stays
                if (it + 1 >= iters) break;  // only c is wanted from here on
            }
            // ---- r = x - q or r -= alpha q; x and y of W^T r
            float4 rg[16];
            if (it < 0) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 *row =
                        reinterpret_cast<const float4 *>(ref.f->data + row_offset(ref, lane, warp + 16 * h));
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float4 x = __ldg(row + k);
                        q[h][4 * k] = x.x - q[h][4 * k];
                        q[h][4 * k + 1] = x.y - q[h][4 * k + 1];
                        q[h][4 * k + 2] = x.z - q[h][4 * k + 2];
                        q[h][4 * k + 3] = x.w - q[h][4 * k + 3];
                    }
                }
            } else {
#pragma unroll
                for (int at = kRShared; at < 16; ++at) rg[at] = Rv[at * kNT];
#pragma unroll
                for (int at = 0; at < 16; ++at) {
                    const int h = at / 8, k = at % 8;
                    const float4 r = at < kRShared ? Rs[at * kNT] : rg[at];
                    q[h][4 * k] = __fmaf_rn(-alpha, q[h][4 * k], r.x);
                    q[h][4 * k + 1] = __fmaf_rn(-alpha, q[h][4 * k + 1], r.y);
                    q[h][4 * k + 2] = __fmaf_rn(-alpha, q[h][4 * k + 2], r.z);
                    q[h][4 * k + 3] = __fmaf_rn(-alpha, q[h][4 * k + 3], r.w);
                }
            }
#pragma unroll
            for (int at = 0; at < 16; ++at) {
                const int h = at / 8, k = at % 8;
                const float4 r = make_float4(q[h][4 * k], q[h][4 * k + 1], q[h][4 * k + 2], q[h][4 * k + 3]);
                if (at < kRShared) Rs[at * kNT] = r;
                else Rv[at * kNT] = r;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) plane_adj<KIND>(sb, warp + 16 * h, q[h]);
            __syncthreads();
            asm volatile("" : "+r"(kp.z[0]), "+r"(kp.z[1]), "+r"(kp.y), "+r"(kp.x[0]), "+r"(kp.x[1]));
            z_adj<KIND, true>(sb, kp);
            // ---- gamma = ||s||^2, s = M W^T r: 4 entries along x at a time
            acc = 0.f;
#pragma unroll 8
            for (int i = 0; i < 16; ++i) {
                const int a = pad_of(4 * tid) + i * (4 * kNT / 1024) * SZ;
                const float v0 = sb[a], v1 = sb[a + 1], v2 = sb[a + 2], v3 = sb[a + 3];
                acc = __fmaf_rn(v0, v0, __fmaf_rn(v1, v1, __fmaf_rn(v2, v2, __fmaf_rn(v3, v3, acc))));
            }
            block_sum(acc, part, [&](double gnew) {
                if (lane == 0) {
                    s_ratio = it < 0 ? 0.f : (float)(gnew / s_gamma);
                    s_gamma = gnew;
                    s_go = gnew > 0.0;
                }
            });
            beta = s_ratio;
            mode = it < 0 ? kFirst : kStep;
            if (!s_go || it + 1 >= iters) break;
        }
        // ---- the refit survivors go out under the plain mask
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int base = pidx(lane, warp + 16 * h, 0);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int at = (8 * h + k) * kNT;
                float4 c = Cv[at];
                if (pending) {
                    const float4 p = Pv[at];
                    c.x = __fmaf_rn(alpha, p.x, c.x);
                    c.y = __fmaf_rn(alpha, p.y, c.y);
                    c.z = __fmaf_rn(alpha, p.z, c.z);
                    c.w = __fmaf_rn(alpha, p.w, c.w);
                }
                sb[base + (4 * k) * SZ] = c.x;
                sb[base + (4 * k + 1) * SZ] = c.y;
                sb[base + (4 * k + 2) * SZ] = c.z;
                sb[base + (4 * k + 3) * SZ] = c.w;
            }
        }
        __syncthreads();
        emit_record(s, g, zmask, shuffle, stage, rec_bytes, chunks);
    }
}

}  // namespace cz

using namespace cz;

namespace {
template <class K>
cudaError_t prep(K kernel, int bytes)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}
constexpr int kDenseSmem = kPadFloats * 4;
}  // namespace

size_t cz_refit_scratch_floats(int grid) { return (size_t)grid * 3 * kBS3; }

cudaError_t cz_launch_iwt_linear(int wtype, const float *coef, float *out, long long nblocks, int grid, cudaStream_t st)
{
    if (nblocks <= 0) return cudaSuccess;
    cudaError_t e;
    switch (wkind(wtype)) {
    case 1:
        if ((e = prep(iwt_linear_kernel<1>, kDenseSmem)) != cudaSuccess) return e;
        iwt_linear_kernel<1><<<grid, kNT, kDenseSmem, st>>>(coef, out, nblocks);
        break;
    case 2:
        if ((e = prep(iwt_linear_kernel<2>, kDenseSmem)) != cudaSuccess) return e;
        iwt_linear_kernel<2><<<grid, kNT, kDenseSmem, st>>>(coef, out, nblocks);
        break;
    default:
        if ((e = prep(iwt_linear_kernel<3>, kDenseSmem)) != cudaSuccess) return e;
        iwt_linear_kernel<3><<<grid, kNT, kDenseSmem, st>>>(coef, out, nblocks);
    }
    return cudaGetLastError();
}

cudaError_t cz_launch_iwt_adjoint(int wtype, const float *in, float *coef, long long nblocks, int grid, cudaStream_t st)
{
    if (nblocks <= 0) return cudaSuccess;
    cudaError_t e;
    switch (wkind(wtype)) {
    case 1:
        if ((e = prep(iwt_adjoint_kernel<1>, kDenseSmem)) != cudaSuccess) return e;
        iwt_adjoint_kernel<1><<<grid, kNT, kDenseSmem, st>>>(in, coef, nblocks);
        break;
    case 2:
        if ((e = prep(iwt_adjoint_kernel<2>, kDenseSmem)) != cudaSuccess) return e;
        iwt_adjoint_kernel<2><<<grid, kNT, kDenseSmem, st>>>(in, coef, nblocks);
        break;
    default:
        if ((e = prep(iwt_adjoint_kernel<3>, kDenseSmem)) != cudaSuccess) return e;
        iwt_adjoint_kernel<3><<<grid, kNT, kDenseSmem, st>>>(in, coef, nblocks);
    }
    return cudaGetLastError();
}

cudaError_t cz_launch_refit(int wtype, const CzField *fields, int nfields, long long total_blocks, int zerobits,
                            int shuffle, int iters, uint8_t *stage, int *rec_bytes, unsigned long long *queue,
                            float *scratch, int grid, cudaStream_t st, CzChunks chunks)
{
    if (total_blocks <= 0) return cudaSuccess;
    const int smem = kRefitSmem;
    cudaError_t e;
    switch (wkind(wtype)) {
    case 1:
        if ((e = prep(refit_kernel<1>, smem)) != cudaSuccess) return e;
        refit_kernel<1><<<grid, kNT, smem, st>>>(fields, nfields, total_blocks, zerobits, shuffle, iters, stage,
                                                 rec_bytes, queue, scratch, chunks);
        break;
    case 2:
        if ((e = prep(refit_kernel<2>, smem)) != cudaSuccess) return e;
        refit_kernel<2><<<grid, kNT, smem, st>>>(fields, nfields, total_blocks, zerobits, shuffle, iters, stage,
                                                 rec_bytes, queue, scratch, chunks);
        break;
    default:
        if ((e = prep(refit_kernel<3>, smem)) != cudaSuccess) return e;
        refit_kernel<3><<<grid, kNT, smem, st>>>(fields, nfields, total_blocks, zerobits, shuffle, iters, stage,
                                                 rec_bytes, queue, scratch, chunks);
    }
    return cudaGetLastError();
}
