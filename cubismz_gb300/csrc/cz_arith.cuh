// cz_arith.cuh -- bit-exact evaluation of the reference's wavelet stencils
// without binary64 arithmetic.
//
// The reference evaluates every stencil in binary64 and rounds to binary32 on
// return: `5./16 * f0 + 15./16 * f1 - 5./16 * f2 + 1./16 * f3` with float
// arguments and a float return type (WaveletsOnInterval.h:33-83). GB300 runs
// binary64 at a small fraction of its binary32 rate, so the kernels compute
// the same bits in binary32:
//
//   * A stencil is sum_i (k_i/D) * v_i with small integers k_i and D in
//     {8,16}. Every product is exact in binary64; whenever the exponents of
//     the inputs are within a bounded spread, every binary64 partial sum is
//     exact too, so the reference result is RN32(exact sum).
//   * Each input v is split against a line-wide grid U = 2^(E+1-B), E being
//     the exponent of the largest input of the line: v = hi + lo with
//     hi = RN_U(v) (two adds with the constant 1.5*2^(E+24-B)) and
//     lo = v - hi, both exact. The hi parts are integers times U of at most
//     2^B, so sum (k/D)*hi is exact in binary32 while K*2^B <= 2^24
//     (K = sum|k_i|). The lo parts are multiples of the smallest input ulp
//     and at most U/2, so sum (k/D)*lo is exact while
//     E - e_min <= B + 1 - log2(K). One final rounded add gives
//     RN32(exact sum). Grids and spreads per stencil are listed below.
//   * Lines whose spread is wider, or whose values sit near the ends of the
//     binary32 range, take the per-stencil path: the same split against the
//     stencil's own maximum, and binary64 only when even that is too wide.
//
// Signed zeros follow the binary64 chain, whose zero is -0 only where all its
// products are: -0 under every positive coefficient, +0 under every negative
// one. That costs no instruction. The result is lo - (-hi): a hi sum that
// vanishes comes out as -hi = +0 (every stencil has coefficients of both signs),
// so the result is the lo sum, whose zeros have the signs of its sources'. Only
// where sources that are not zero cancel would their lo (+0) pass for a zero
// source's; that takes two sources of one coefficient sign, so it concerns W1M
// and W1L (see there). A line with a -0 thus needs no path of its own: a field with
// a -0 background takes the encode kernel 61 us at 256^3; with such lines on the
// out-of-line path below it took 172.
//
// What bounds a line on the GPU is instruction issue, so the main path keeps
// (hi, lo) as a register pair and evaluates both chains with packed binary32
// arithmetic (two roundings per instruction, each as the scalar one's):
// 5 instructions per 4-point stencil instead of 10; and it finds the line's
// largest and smallest non-zero magnitude with three-input minima and maxima,
// 2 instructions per source instead of 4. Encode kernel at 512^3: 0.516 -> 0.416
// ms (wtype 1). The other paths are rare and stay out of line, which keeps the
// kernels' code small.
//
// All binary32 arithmetic goes through explicit round-to-nearest intrinsics so
// the compiler cannot contract or reassociate it; host builds use
// -ffp-contract=off and the C99 fmaf.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define CZ_HD __host__ __device__ __forceinline__
#define CZ_RARE static __host__ __device__ __noinline__
#else
#include <math.h>
#include <string.h>
#define CZ_HD static inline
#define CZ_RARE static inline
#endif

#if defined(__CUDA_ARCH__)
#define CZ_FMA(a, b, c) __fmaf_rn((a), (b), (c))
#define CZ_ADD(a, b) __fadd_rn((a), (b))
#define CZ_SUB(a, b) __fsub_rn((a), (b))
#define CZ_MUL(a, b) __fmul_rn((a), (b))
#define CZ_DMUL(a, b) __dmul_rn((a), (b))
#define CZ_DFMA(a, b, c) __fma_rn((a), (b), (c))
#define CZ_D2F(a) __double2float_rn(a)
#define CZ_BITS(x) __float_as_uint(x)
#define CZ_FLT(u) __uint_as_float(u)
#define CZ_UMIN(a, b) min((a), (b))
#define CZ_UMAX(a, b) max((a), (b))
#else
#define CZ_FMA(a, b, c) fmaf((a), (b), (c))
#define CZ_ADD(a, b) ((float)((a) + (b)))
#define CZ_SUB(a, b) ((float)((a) - (b)))
#define CZ_MUL(a, b) ((float)((a) * (b)))
#define CZ_DMUL(a, b) ((double)(a) * (double)(b))
#define CZ_DFMA(a, b, c) fma((a), (b), (c))
#define CZ_D2F(a) ((float)(a))
CZ_HD uint32_t cz_bits_h(float x)
{
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
}
CZ_HD float cz_flt_h(uint32_t u)
{
    float x;
    memcpy(&x, &u, 4);
    return x;
}
#define CZ_BITS(x) cz_bits_h(x)
#define CZ_FLT(u) cz_flt_h(u)
#define CZ_UMIN(a, b) ((a) < (b) ? (a) : (b))
#define CZ_UMAX(a, b) ((a) > (b) ? (a) : (b))
#endif

namespace cz {

// Split grids and spreads. A line's sources are split against U = 2^(E+1-B)
// (E: exponent of the line maximum). Exactness needs, for a stencil with
// coefficient sum K = sum|k_i|:
//   hi sums:  K * 2^B <= 2^24
//   lo sums:  E - e_min <= B + 1 - log2(K)   (e_min: smallest non-zero input)
// B = 19 serves every stencil with K <= 32 with a spread of 15 binades
// (interp first/middle/one-to-last: K = 26/20/26; average-interpolating
// predictors: K <= 16). interp_last (K = 96) is re-split on B = 17, spread 11.
constexpr int kGridBits = 19;
constexpr int kSpread = 15;
constexpr int kLastGridBits = 17;
constexpr int kLastSpread = 11;

// Stencil coefficient sets k/D, exactly representable in binary32.
// WaveletsOnInterval.h:33-51 (D = 16) and :55-83 (D = 8).
struct W1F { static constexpr float c[4] = {5.f / 16, 15.f / 16, -5.f / 16, 1.f / 16}; };
struct W1M { static constexpr float c[4] = {-1.f / 16, 9.f / 16, 9.f / 16, -1.f / 16}; };
struct W1O { static constexpr float c[4] = {1.f / 16, -5.f / 16, 15.f / 16, 5.f / 16}; };
struct W1L { static constexpr float c[4] = {-5.f / 16, 21.f / 16, -35.f / 16, 35.f / 16}; };
struct P0F { static constexpr float c[3] = {11.f / 8, -1.f / 2, 1.f / 8}; };
struct P1F { static constexpr float c[3] = {5.f / 8, 1.f / 2, -1.f / 8}; };
struct P0M { static constexpr float c[3] = {1.f / 8, 1.f, -1.f / 8}; };
struct P1M { static constexpr float c[3] = {-1.f / 8, 1.f, 1.f / 8}; };
struct P0L { static constexpr float c[3] = {-1.f / 8, 1.f / 2, 5.f / 8}; };
struct P1L { static constexpr float c[3] = {1.f / 8, -1.f / 2, 11.f / 8}; };

// Exponent analysis of a set of stencil sources: biased exponent of the
// largest magnitude, and whether every non-zero source lies within `spread`
// binades of it (with the range limits that keep all grids representable:
// 27 <= eb keeps every grid at or above 2^-149, eb <= 247 keeps the split
// constants finite; an all-zero set is exact with any constant).
template <int H>
CZ_HD uint32_t max_bits(const float (&v)[H])
{
    uint32_t amax = 0;
#pragma unroll
    for (int i = 0; i < H; ++i) amax = CZ_UMAX(amax, CZ_BITS(v[i]) & 0x7fffffffu);
    return amax;
}
template <int H>
CZ_HD bool within(const float (&v)[H], uint32_t amax, int spread)
{
    const uint32_t eb = amax >> 23;
    // non-zero |v| below 2^(E-spread)  <=>  (bits-1) < (threshold bits - 1)
    const uint32_t tb = ((eb - (uint32_t)spread) << 23) - 1u;
    uint32_t small = 0;
#pragma unroll
    for (int i = 0; i < H; ++i) small |= (uint32_t)(((CZ_BITS(v[i]) & 0x7fffffffu) - 1u) < tb);
    return (amax == 0u) || (eb >= 27u && eb <= 247u && !small);
}

// Split constant 1.5*2^(E+24-B); its ulp is the grid U = 2^(E+1-B).
template <int B>
CZ_HD float split_const(uint32_t amax)
{
    const uint32_t eb = amax == 0u ? 127u : CZ_UMIN(CZ_UMAX(amax >> 23, 27u), 247u);
    return CZ_FLT(((eb + (uint32_t)(24 - B)) << 23) | 0x400000u);
}

template <int H>
CZ_HD void split(const float (&v)[H], float C, float (&hi)[H], float (&lo)[H])
{
#pragma unroll
    for (int i = 0; i < H; ++i) {
        hi[i] = CZ_SUB(CZ_ADD(v[i], C), C);
        lo[i] = CZ_SUB(v[i], hi[i]);
    }
}

// Minimum of three.
CZ_HD uint32_t umin3(uint32_t a, uint32_t b, uint32_t c)
{
#if defined(__CUDA_ARCH__)
    return __vimin3_u32(a, b, c);
#else
    return CZ_UMIN(CZ_UMIN(a, b), c);
#endif
}
// Largest magnitude of three, a NaN if one of them is.
CZ_HD float amax3(float a, float b, float c)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    const uint32_t x = CZ_BITS(a) & 0x7fffffffu, y = CZ_BITS(b) & 0x7fffffffu, z = CZ_BITS(c) & 0x7fffffffu;
    return CZ_FLT(CZ_UMAX(CZ_UMAX(x, y), z));
#endif
}

// Whether the split grids are exact for sources of largest magnitude amax and
// smallest non-zero magnitude lo2 (as 2 bits - 1, which orders the non-zero
// magnitudes and puts zeros past them all): all non-zero ones within `spread`
// binades of the largest, and that one within the grids' range (or everything
// zero).
CZ_HD bool in_range(uint32_t amax, uint32_t lo2, int spread)
{
    const uint32_t eb = CZ_UMIN(CZ_UMAX(amax >> 23, 27u), 247u);
    return (amax == 0u || (amax >> 23) == eb) && lo2 >= ((eb - (uint32_t)spread) << 24) - 1u;
}

// Exponent analysis of a line's sources (H even). Returns whether the main
// path is exact for every stencil with K <= 32 on this line. `narrow`: the last
// four, which interp_last takes, lie within kLastSpread binades of the largest
// (noise-like sources: all but one line in 170; for all 16 of them it would be
// one in 40).
template <int H>
CZ_HD bool line_grid(const float (&v)[H], uint32_t &amax, bool &narrow)
{
    auto x = [&](int i) { return 2u * CZ_BITS(v[i]) - 1u; };
    float m = amax3(v[0], v[1], v[1]);
    const uint32_t last = umin3(CZ_UMIN(x(H - 4), x(H - 3)), x(H - 2), x(H - 1));
    uint32_t lo = last;
#pragma unroll
    for (int i = 2; i < H; i += 2) m = amax3(m, v[i], v[i + 1]);
#pragma unroll
    for (int i = 0; i < H - 4; i += 2) lo = umin3(lo, x(i), x(i + 1));
    amax = CZ_BITS(m);
    const uint32_t eb = CZ_UMIN(CZ_UMAX(amax >> 23, 27u), 247u);
    narrow = last >= ((eb - (uint32_t)kLastSpread) << 24) - 1u;
    return (amax == 0u || (amax >> 23) == eb) && lo >= ((eb - (uint32_t)kSpread) << 24) - 1u;
}

// Line-level analysis and split on the main grid.
template <int H>
CZ_HD bool line_split(const float (&v)[H], float (&hi)[H], float (&lo)[H], uint32_t &amax)
{
    bool narrow;
    const bool ok = line_grid<H>(v, amax, narrow);
    split<H>(v, split_const<kGridBits>(amax), hi, lo);
    return ok;
}

// A pair of hi (or -hi) and lo, and packed binary32 arithmetic on it.
struct Pair {
#if defined(__CUDA_ARCH__)
    unsigned long long v;
#else
    float a, b;
#endif
};
CZ_HD Pair pair(float a, float b)
{
    Pair p;
#if defined(__CUDA_ARCH__)
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
#else
    p.a = a;
    p.b = b;
#endif
    return p;
}
CZ_HD Pair pmul(Pair x, Pair y)
{
    Pair p;
#if defined(__CUDA_ARCH__)
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(x.v), "l"(y.v));
#else
    p.a = CZ_MUL(x.a, y.a);
    p.b = CZ_MUL(x.b, y.b);
#endif
    return p;
}
CZ_HD Pair pfma(Pair x, Pair y, Pair z)
{
    Pair p;
#if defined(__CUDA_ARCH__)
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(x.v), "l"(y.v), "l"(z.v));
#else
    p.a = CZ_FMA(x.a, y.a, z.a);
    p.b = CZ_FMA(x.b, y.b, z.b);
#endif
    return p;
}
CZ_HD Pair padd(Pair x, Pair y)
{
    Pair p;
#if defined(__CUDA_ARCH__)
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(x.v), "l"(y.v));
#else
    p.a = CZ_ADD(x.a, y.a);
    p.b = CZ_ADD(x.b, y.b);
#endif
    return p;
}
// The sum rounded down: exact operands, so only its zeros differ (-0 unless
// both are +0).
CZ_HD Pair padd_rd(Pair x, Pair y)
{
    Pair p;
#if defined(__CUDA_ARCH__)
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(p.v) : "l"(x.v), "l"(y.v));
#else
    p.a = CZ_ADD(x.a, y.a);
    p.b = CZ_ADD(x.b, y.b);
    if (p.a == 0.f) p.a = CZ_BITS(x.a) | CZ_BITS(y.a) ? -0.f : 0.f;
    if (p.b == 0.f) p.b = CZ_BITS(x.b) | CZ_BITS(y.b) ? -0.f : 0.f;
#endif
    return p;
}
CZ_HD Pair pfma_rd(Pair x, Pair y, Pair z)
{
    Pair p;
#if defined(__CUDA_ARCH__)
    asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(p.v) : "l"(x.v), "l"(y.v), "l"(z.v));
#else
    p = padd_rd(pmul(x, y), z);
#endif
    return p;
}
CZ_HD void unpair(Pair x, float &a, float &b)
{
#if defined(__CUDA_ARCH__)
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
#else
    a = x.a;
    b = x.b;
#endif
}
// hi + lo of a chain's (-hi, lo).
CZ_HD float psum(Pair x)
{
    float a, b;
    unpair(x, a, b);
    return CZ_SUB(b, a);
}
CZ_HD Pair split_pair(float v, float C)
{
    const float hi = CZ_SUB(CZ_ADD(v, C), C);
    return pair(hi, CZ_SUB(v, hi));
}
// (-hi, lo): -hi rounded down, which is exact, and -0 where it vanishes.
CZ_HD Pair split_neg(float v, float C)
{
#if defined(__CUDA_ARCH__)
    const float n = __fsub_rd(C, CZ_ADD(v, C));
#else
    float n = CZ_SUB(C, CZ_ADD(v, C));
    if (n == 0.f) n = -0.f;
#endif
    return pair(n, CZ_ADD(v, n));
}
// RN32 of sum c_i*(hi_i+lo_i) given an exact split (see header): the
// interpolating stencils from (hi, lo), the averaging ones from (-hi, lo), whose
// middle has no product to negate hi with.
template <class S>
CZ_HD float st4_pair(Pair p0, Pair p1, Pair p2, Pair p3)
{
    constexpr float k0 = S::c[0], k1 = S::c[1], k2 = S::c[2], k3 = S::c[3];
    return psum(pfma(pair(-k3, k3), p3, pfma(pair(-k2, k2), p2, pfma(pair(-k1, k1), p1, pmul(pair(-k0, k0), p0)))));
}
template <class S>
CZ_HD float st3_pair(Pair p0, Pair p1, Pair p2)
{
    constexpr float k0 = S::c[0], k1 = S::c[1], k2 = S::c[2];
    return psum(pfma(pair(k2, k2), p2, pfma(pair(k1, k1), p1, pmul(pair(k0, k0), p0))));
}
// The two interpolating stencils with two negative coefficients: from u and w,
// the exact sums of what is added and of what is taken away, u - w. w is rounded
// down: its lo is +0 only where both its sources are, its hi -0 only where two
// that are not zero cancel, which makes the zero +0 again. Here:
// 16 times W1M, RN32 of 9 (p1 + p2) - (p0 + p3). Scaling by a power of two
// commutes with the rounding (line_grid keeps a line's sums clear of the
// subnormals), so the caller's fma with 1/16 gives the bits of the stencil's
// own rounding followed by the add. 8 cycles of the fma pipe instead of the
// chain's 10.
CZ_HD float w1m_16(Pair p0, Pair p1, Pair p2, Pair p3)
{
    float uh, ul, wh, wl;
    unpair(padd(p1, p2), uh, ul);
    unpair(padd_rd(p0, p3), wh, wl);
    return CZ_SUB(CZ_FMA(9.f, ul, -wl), CZ_FMA(-9.f, uh, wh));
}
CZ_HD float w1l(Pair p0, Pair p1, Pair p2, Pair p3)
{
    constexpr float k0 = -W1L::c[0], k1 = W1L::c[1], k2 = -W1L::c[2], k3 = W1L::c[3];
    float uh, ul, wh, wl;
    unpair(pfma(pair(k3, k3), p3, pmul(pair(k1, k1), p1)), uh, ul);
    unpair(pfma_rd(pair(k2, k2), p2, pmul(pair(k0, k0), p0)), wh, wl);
    return CZ_SUB(CZ_SUB(ul, wl), CZ_SUB(wh, uh));
}
// Stencils on the grid of split constant C.
template <class S>
CZ_HD float st4_on(float v0, float v1, float v2, float v3, float C)
{
    return st4_pair<S>(split_pair(v0, C), split_pair(v1, C), split_pair(v2, C), split_pair(v3, C));
}
CZ_HD float w1m_on(float v0, float v1, float v2, float v3, float C)
{
    return 0.0625f * w1m_16(split_pair(v0, C), split_pair(v1, C), split_pair(v2, C), split_pair(v3, C));
}
CZ_HD float w1l_on(float v0, float v1, float v2, float v3, float C)
{
    return w1l(split_pair(v0, C), split_pair(v1, C), split_pair(v2, C), split_pair(v3, C));
}
// The P0M and P1M stencils: p1 +- (p0 - p2) / 8. The difference is -0 where p0
// is -0 and p2 is +0, as P0M's products are; rounded down, +0 where P1M's are.
CZ_HD void avg_mid(Pair p0, Pair p1, Pair p2, float &even, float &odd)
{
    const Pair m = pair(-1.f, -1.f), t = pfma(m, p2, p0), u = pfma_rd(m, p2, p0);
    even = psum(pfma(pair(0.125f, 0.125f), t, p1));
    odd = psum(pfma(pair(-0.125f, -0.125f), u, p1));
}

// The reference arithmetic itself: binary64 products summed left to right,
// rounded to binary32 once (used when no exact binary32 split exists). The
// products are exact, so an fma rounds like the sum alone.
template <class S>
CZ_HD float st4_f64(float v0, float v1, float v2, float v3)
{
    constexpr double k0 = S::c[0], k1 = S::c[1], k2 = S::c[2], k3 = S::c[3];
    return CZ_D2F(CZ_DFMA(k3, (double)v3, CZ_DFMA(k2, (double)v2, CZ_DFMA(k1, (double)v1, CZ_DMUL(k0, (double)v0)))));
}
template <class S>
CZ_HD float st3_f64(float v0, float v1, float v2)
{
    constexpr double k0 = S::c[0], k1 = S::c[1], k2 = S::c[2];
    return CZ_D2F(CZ_DFMA(k2, (double)v2, CZ_DFMA(k1, (double)v1, CZ_DMUL(k0, (double)v0))));
}

// Per-stencil path: the stencil's own grid, or binary64.
template <class S>
CZ_HD float st4_any(float v0, float v1, float v2, float v3)
{
    const float v[4] = {v0, v1, v2, v3};
    const uint32_t amax = max_bits<4>(v);
    if (within<4>(v, amax, kSpread)) return st4_on<S>(v0, v1, v2, v3, split_const<kGridBits>(amax));
    return st4_f64<S>(v0, v1, v2, v3);
}
template <class S>
CZ_HD float st3_any(float v0, float v1, float v2)
{
    const float v[3] = {v0, v1, v2};
    const uint32_t amax = max_bits<3>(v);
    if (within<3>(v, amax, kSpread)) {
        const float C = split_const<kGridBits>(amax);
        return st3_pair<S>(split_neg(v0, C), split_neg(v1, C), split_neg(v2, C));
    }
    return st3_f64<S>(v0, v1, v2);
}

// interp_last on a line's last four sources (K = 96, its own coarser grid),
// given the line maximum; `narrow` as line_grid says. Otherwise their own
// maximum's grid, or binary64.
CZ_RARE float interp_last_wide(float v0, float v1, float v2, float v3)
{
    const float v[4] = {v0, v1, v2, v3};
    const uint32_t amax = max_bits<4>(v);
    if (within<4>(v, amax, kLastSpread)) return w1l_on(v0, v1, v2, v3, split_const<kLastGridBits>(amax));
    return st4_f64<W1L>(v0, v1, v2, v3);
}
CZ_HD float interp_last(float v0, float v1, float v2, float v3, uint32_t line_amax, bool narrow)
{
    if (!narrow) return interp_last_wide(v0, v1, v2, v3);
    return w1l_on(v0, v1, v2, v3, split_const<kLastGridBits>(line_amax));
}

}  // namespace cz
