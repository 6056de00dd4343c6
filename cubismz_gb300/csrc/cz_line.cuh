// cz_line.cuh -- one 1D interval-wavelet transform of a line held in
// registers, bit-exact to WI4::transform<N,forward> (WaveletsOnInterval.h:85-201).
//
// Layout of a transformed line: [N/2 scalings | N/2 details] along the line.
// wtype 1: 4th-order interpolating; 2: the same with the lifting update of the
// scalings; any other value: 3rd-order average-interpolating (the reference
// treats wtype 0 and 3 alike, :154).
#pragma once
#include "cz_arith.cuh"

namespace cz {

// ---------------------------------------------------------------- wtype 1/2
// Predictions of a line's odd samples from its H scalings e
// (WaveletsOnInterval.h:33-51) where one grid does not do for the line: every
// four neighbours on a grid of their own, binary64 where even that is not exact.
// Out of line and rolled, one prediction after the other: noise has a few such
// lines, and unrolled whole it took more from the kernels' other code (encode at
// 512^3 0.429 ms instead of 0.417) than it gave where most lines come here. Fields
// whose lines come here, 256^3, encode kernel: a volume fraction's interface
// (1 to 6e-8) 113 us, a wide Gaussian 462; 115 and 573 unrolled in place with a
// grid per prediction.
CZ_RARE void interp_wide(const float *__restrict__ e, float *__restrict__ o, int H)
{
    float v0 = e[0], v1 = e[1], v2 = e[2], v3 = e[3];
    o[0] = st4_any<W1F>(v0, v1, v2, v3);
#pragma unroll 1
    for (int i = 1;; ++i) {
        const uint32_t amax = CZ_BITS(amax3(v0, v1, amax3(v2, v3, v3)));
        const uint32_t lo = umin3(2u * CZ_BITS(v0) - 1u, 2u * CZ_BITS(v1) - 1u,
                                  CZ_UMIN(2u * CZ_BITS(v2) - 1u, 2u * CZ_BITS(v3) - 1u));
        float r = w1m_on(v0, v1, v2, v3, split_const<kGridBits>(amax));
        if (!in_range(amax, lo, kSpread)) r = st4_f64<W1M>(v0, v1, v2, v3);
        o[i] = r;
        if (i == H - 3) break;
        v0 = v1;
        v1 = v2;
        v2 = v3;
        v3 = e[i + 3];
    }
    o[H - 2] = st4_any<W1O>(v0, v1, v2, v3);
    o[H - 1] = interp_last_wide(v0, v1, v2, v3);
}
// o[i] = base[i] + sign * prediction i, each rounded as the reference rounds
// (the prediction, then the sum).
template <int H>
CZ_HD void interp_predict(const float (&e)[H], float sign, const float (&base)[H], float (&o)[H])
{
    uint32_t amax;
    bool narrow;
    if (line_grid<H>(e, amax, narrow)) {
        const float C = split_const<kGridBits>(amax);
        Pair p[H];
#pragma unroll
        for (int i = 0; i < H; ++i) p[i] = split_pair(e[i], C);
        o[0] = CZ_FMA(sign, st4_pair<W1F>(p[0], p[1], p[2], p[3]), base[0]);
#pragma unroll
        for (int i = 1; i < H - 2; ++i)
            o[i] = CZ_FMA(0.0625f * sign, w1m_16(p[i - 1], p[i], p[i + 1], p[i + 2]), base[i]);
        o[H - 2] = CZ_FMA(sign, st4_pair<W1O>(p[H - 4], p[H - 3], p[H - 2], p[H - 1]), base[H - 2]);
        o[H - 1] = CZ_FMA(sign, interp_last(e[H - 4], e[H - 3], e[H - 2], e[H - 1], amax, narrow), base[H - 1]);
    } else {
        float te[H], to[H];  // the call's arrays live in memory, e and o in registers
#pragma unroll
        for (int i = 0; i < H; ++i) te[i] = e[i];
        interp_wide(te, to, H);
#pragma unroll
        for (int i = 0; i < H; ++i) o[i] = CZ_FMA(sign, to[i], base[i]);
    }
}

template <int N>
CZ_HD void fwd_interp(float (&x)[N], bool lifting)
{
    constexpr int H = N / 2;
    float e[H], b[H], d[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        e[i] = x[2 * i];
        b[i] = x[2 * i + 1];
    }
    interp_predict<H>(e, -1.f, b, d);
    // scalings[i] += 0.5*details[i] in binary64, rounded to binary32 (:124-126):
    // a single fma is the correctly rounded value of the same exact sum.
#pragma unroll
    for (int i = 0; i < H; ++i) x[i] = lifting ? CZ_FMA(0.5f, d[i], e[i]) : e[i];
#pragma unroll
    for (int i = 0; i < H; ++i) x[H + i] = d[i];
}

template <int N>
CZ_HD void inv_interp(float (&x)[N], bool lifting)
{
    constexpr int H = N / 2;
    float s[H], d[H], o[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        d[i] = x[H + i];
        s[i] = lifting ? CZ_FMA(-0.5f, d[i], x[i]) : x[i];  // :137-139
    }
    interp_predict<H>(s, 1.f, d, o);
    // :141-151: even samples are the scalings, odd samples interp + detail
#pragma unroll
    for (int i = 0; i < H; ++i) {
        x[2 * i] = s[i];
        x[2 * i + 1] = o[i];
    }
}

// ---------------------------------------------------------------- wtype 3
// Predictions of a line's even and odd samples from its H scalings s
// (WaveletsOnInterval.h:55-83), as interp_wide: every three neighbours on a grid
// of their own.
CZ_RARE void avg_wide(const float *__restrict__ s, float *__restrict__ o0, float *__restrict__ o1, int H)
{
    float v0 = s[0], v1 = s[1], v2 = s[2];
    o0[0] = st3_any<P0F>(v0, v1, v2);
    o1[0] = st3_any<P1F>(v0, v1, v2);
#pragma unroll 1
    for (int i = 1;; ++i) {
        const uint32_t amax = CZ_BITS(amax3(v0, v1, v2));
        const uint32_t lo = umin3(2u * CZ_BITS(v0) - 1u, 2u * CZ_BITS(v1) - 1u, 2u * CZ_BITS(v2) - 1u);
        const float C = split_const<kGridBits>(amax);
        float even, odd;
        avg_mid(split_neg(v0, C), split_neg(v1, C), split_neg(v2, C), even, odd);
        if (!in_range(amax, lo, kSpread)) {
            even = st3_f64<P0M>(v0, v1, v2);
            odd = st3_f64<P1M>(v0, v1, v2);
        }
        o0[i] = even;
        o1[i] = odd;
        if (i == H - 2) break;
        v0 = v1;
        v1 = v2;
        v2 = s[i + 2];
    }
    o0[H - 1] = st3_any<P0L>(v0, v1, v2);
    o1[H - 1] = st3_any<P1L>(v0, v1, v2);
}
template <int H>
CZ_HD void avg_predict(const float (&s)[H], float (&p0)[H], float (&p1)[H])
{
    uint32_t amax;
    bool narrow;
    if (line_grid<H>(s, amax, narrow)) {
    const float C = split_const<kGridBits>(amax);
    Pair p[H];
#pragma unroll
    for (int i = 0; i < H; ++i) p[i] = split_neg(s[i], C);
    p0[0] = st3_pair<P0F>(p[0], p[1], p[2]);
    p1[0] = st3_pair<P1F>(p[0], p[1], p[2]);
#pragma unroll
    for (int i = 1; i < H - 1; ++i) avg_mid(p[i - 1], p[i], p[i + 1], p0[i], p1[i]);
    p0[H - 1] = st3_pair<P0L>(p[H - 3], p[H - 2], p[H - 1]);
    p1[H - 1] = st3_pair<P1L>(p[H - 3], p[H - 2], p[H - 1]);
    } else {
        float t[H], t0[H], t1[H];  // the call's arrays live in memory
#pragma unroll
        for (int i = 0; i < H; ++i) t[i] = s[i];
        avg_wide(t, t0, t1, H);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            p0[i] = t0[i];
            p1[i] = t1[i];
        }
    }
}

template <int N>
CZ_HD void fwd_avg(float (&x)[N])
{
    constexpr int H = N / 2;
    float s[H], d[H], p0[H], p1[H];
    // scalings = 0.5*(x0+x1): binary32 add, exact halving (:159-160)
#pragma unroll
    for (int i = 0; i < H; ++i) s[i] = CZ_MUL(0.5f, CZ_ADD(x[2 * i], x[2 * i + 1]));
    avg_predict<H>(s, p0, p1);
    // details = 0.5*((x1-x0) - (p1-p0)), every step in binary32 (:164-176)
#pragma unroll
    for (int i = 0; i < H; ++i)
        d[i] = CZ_MUL(0.5f, CZ_SUB(CZ_SUB(x[2 * i + 1], x[2 * i]), CZ_SUB(p1[i], p0[i])));
#pragma unroll
    for (int i = 0; i < H; ++i) {
        x[i] = s[i];
        x[H + i] = d[i];
    }
}

template <int N>
CZ_HD void inv_avg(float (&x)[N])
{
    constexpr int H = N / 2;
    float s[H], d[H], p0[H], p1[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        s[i] = x[i];
        d[i] = x[H + i];
    }
    avg_predict<H>(s, p0, p1);
    // :187-197
#pragma unroll
    for (int i = 0; i < H; ++i) {
        x[2 * i] = CZ_SUB(p0[i], d[i]);
        x[2 * i + 1] = CZ_ADD(p1[i], d[i]);
    }
}

template <int N>
CZ_HD void fwd_line(float (&x)[N], int wtype)
{
    if (wtype == 1 || wtype == 2) fwd_interp<N>(x, wtype == 2);
    else fwd_avg<N>(x);
}
template <int N>
CZ_HD void inv_line(float (&x)[N], int wtype)
{
    if (wtype == 1 || wtype == 2) inv_interp<N>(x, wtype == 2);
    else inv_avg<N>(x);
}

}  // namespace cz
