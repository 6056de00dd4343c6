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
// (WaveletsOnInterval.h:33-51), stencil by stencil.
CZ_RARE void interp_rare(const float *e, float *o, int H)
{
    o[0] = st4_main<W1F>(e[0], e[1], e[2], e[3]);
#pragma unroll 1
    for (int i = 1; i < H - 2; ++i) o[i] = st4_main<W1M>(e[i - 1], e[i], e[i + 1], e[i + 2]);
    o[H - 2] = st4_main<W1O>(e[H - 4], e[H - 3], e[H - 2], e[H - 1]);
    o[H - 1] = st4_lastany(e[H - 4], e[H - 3], e[H - 2], e[H - 1]);
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
        Pair u[H - 1];
#pragma unroll
        for (int i = 0; i < H - 1; ++i) u[i] = padd(p[i], p[i + 1]);
#pragma unroll
        for (int i = 1; i < H - 2; ++i) o[i] = CZ_FMA(0.0625f * sign, w1m_16(u[i - 1], u[i], u[i + 1]), base[i]);
        o[H - 2] = CZ_FMA(sign, st4_pair<W1O>(p[H - 4], p[H - 3], p[H - 2], p[H - 1]), base[H - 2]);
        o[H - 1] = CZ_FMA(sign, interp_last(e[H - 4], e[H - 3], e[H - 2], e[H - 1], amax, narrow), base[H - 1]);
    } else {
        float te[H], to[H];  // the call's arrays live in memory, e and o in registers
#pragma unroll
        for (int i = 0; i < H; ++i) te[i] = e[i];
        interp_rare(te, to, H);
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
// (WaveletsOnInterval.h:55-83).
CZ_RARE void avg_rare(const float *s, float *p0, float *p1, int H)
{
    p0[0] = st3_any<P0F>(s[0], s[1], s[2]);
    p1[0] = st3_any<P1F>(s[0], s[1], s[2]);
#pragma unroll 1
    for (int i = 1; i < H - 1; ++i) {
        p0[i] = st3_any<P0M>(s[i - 1], s[i], s[i + 1]);
        p1[i] = st3_any<P1M>(s[i - 1], s[i], s[i + 1]);
    }
    p0[H - 1] = st3_any<P0L>(s[H - 3], s[H - 2], s[H - 1]);
    p1[H - 1] = st3_any<P1L>(s[H - 3], s[H - 2], s[H - 1]);
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
        for (int i = 0; i < H; ++i) p[i] = split_pair(s[i], C);
        p0[0] = st3_pair<P0F>(p[0], p[1], p[2]);
        p1[0] = st3_pair<P1F>(p[0], p[1], p[2]);
#pragma unroll
        for (int i = 1; i < H - 1; ++i) {
            // p[i] +- (p[i-1] - p[i+1]) / 8: the difference is shared (exact,
            // and +0 where it vanishes)
            const Pair t = pfma(pair(-1.f, -1.f), p[i + 1], p[i - 1]);
            p0[i] = psum(pfma(pair(0.125f, 0.125f), t, p[i]));
            p1[i] = psum(pfma(pair(-0.125f, -0.125f), t, p[i]));
        }
        p0[H - 1] = st3_pair<P0L>(p[H - 3], p[H - 2], p[H - 1]);
        p1[H - 1] = st3_pair<P1L>(p[H - 3], p[H - 2], p[H - 1]);
    } else {
        float t[H], t0[H], t1[H];
#pragma unroll
        for (int i = 0; i < H; ++i) t[i] = s[i];
        avg_rare(t, t0, t1, H);
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
