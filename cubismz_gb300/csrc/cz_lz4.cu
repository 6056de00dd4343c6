// cz_lz4.cu -- LZ4 legacy block format on the GPU.
//
// Encoder: greedy parse, format-compatible with the reference decoder
// LZ4_uncompress_unknownOutputSize (ThirdParty/lz4/lz4.c:802-905): minimum
// match 4, offsets 1..65535, the last 5 bytes are literals and the last
// match starts at least 12 bytes before the end (lz4.c:177-204). A warp
// takes super-windows of 512 or 768 positions (see window_for):
//   * probe  -- 4 positions per lane per step from coalesced word loads; a
//     hash table of 1024 entries per warp in shared memory holds position
//     (mod 2^18) and a 14-bit tag of the 4-byte sequence, so most false
//     candidates are dropped without reading memory;
//   * walk   -- lane k parses its 16 or 24 positions greedily, jumping
//     from one position with a candidate to the next (a bitmask of its
//     candidate slots) and measuring matches against memory;
//   * merge  -- lane k keeps the sequences that start at or after the end
//     of the last kept match of lanes < k (one ballot when no match crosses
//     a later lane's last start, the exact serial rule otherwise);
//   * emit   -- a warp scan places every kept sequence, each lane writes its
//     own; literal runs over 32 bytes are copied by 8 lanes each, from 256 on
//     by the whole warp.
// With few chunks a second warp does the emission while the first parses on
// (lz4_encode_pair_kernel).
// Parse effort (a template level, cz_set_lz4_effort): 1 (default) extends
// kept matches backwards over equal bytes (lz4.c's "catch up") and keeps
// the tail of a match that a lower lane's match overlaps; 2 also takes
// repeats at distance 1-3 that the table misses and starts each lane's
// walk 8 positions early; 0 does neither.
// Windows without a match advance faster after repeated misses (the
// reference's acceleration idea, lz4.c:389-393). Chunks of block records
// ([int32 nbytes][mask][4 byte planes], shuffle on) skip the search over
// byte planes 1 and 2 -- the two middle mantissa bytes, which do not
// compress -- and copy them as literals; those literal bytes are not even
// copied here: the encoder leaves their span of its output unwritten and
// records it per chunk, and the gather that packs the stream copies them
// straight from the records. The same parse in SEQ mode feeds the DEFLATE
// encoder (cz_zlib.cu).
// Decoder: the same acceptance tests and error convention as
// LZ4_uncompress_unknownOutputSize (-(input position) on malformed input; an
// empty input yields 0). Two kernels, chosen by the number of chunks: one
// CTA per chunk for few, one warp per chunk for many. Both parse windows of
// 128 input bytes speculatively (every lane decodes tokens at 4 candidate
// positions; jump tables by pointer doubling find the real sequences) and
// stage output in a ring in shared memory that is flushed with word stores;
// overlapping matches repeat their first `offset` bytes, the byte-serial copy
// semantics. For one-record chunks of shuffled records a literal run that
// covers byte planes 1 and 2 whole stays in the input (hole), where later
// matches and the decode kernel read it.
#include <algorithm>

#include "cz_bytes.cuh"
#include "cz_codec.h"
#include "cz_deflate.cuh"

namespace cz {

constexpr int kHashLog = 10;
constexpr uint32_t kEmpty = 0xffffffffu;
constexpr int kMinMatch = 4, kLastLiterals = 5, kMfLimit = 12;

__device__ __forceinline__ uint32_t lz_hash(uint32_t v) { return (v * 2654435761u) >> (32 - kHashLog); }

__device__ __forceinline__ unsigned lanemask_lt_()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// 32-bit little-endian word at any byte address (two aligned loads).
__device__ __forceinline__ uint32_t rd32u(const uint8_t *p)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t sh = (uint32_t)(a & 3) * 8;
    return sh ? __funnelshift_r(w[0], w[1], sh) : w[0];
}

// 16 bytes at any byte address as four little-endian words: five aligned
// loads, all issued before any use. May read up to 19 bytes past p (inputs
// carry tail room).
__device__ __forceinline__ void rd16u(const uint8_t *p, uint32_t (&v)[4])
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t sh = (uint32_t)(a & 3) * 8;
    uint32_t x[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) x[j] = w[j];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = sh ? __funnelshift_r(x[j], x[j + 1], sh) : x[j];
}

// Warp-wide copy of n bytes; 4-byte stores once dst is aligned. May read up
// to 4 bytes past src+n (inputs carry tail room).
__device__ __forceinline__ void warp_copy(uint8_t *dst, const uint8_t *src, int n, int lane)
{
    int h = (int)((4 - (reinterpret_cast<uintptr_t>(dst) & 3)) & 3);
    if (h > n) h = n;
    if (lane < h) dst[lane] = src[lane];
    dst += h;
    src += h;
    n -= h;
    const int nw = n >> 2;
    const uint32_t sa = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3);
    const uint32_t *sw = reinterpret_cast<const uint32_t *>(src - sa);
    uint32_t *dw = reinterpret_cast<uint32_t *>(dst);
    // 8 words per lane in flight: every load of a round before its stores
    constexpr int U = 8;
    for (int i0 = 0; i0 < nw; i0 += 32 * U) {
        uint32_t v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + 32 * u + lane;
            v[u] = i < nw ? (sa ? __funnelshift_r(sw[i], sw[i + 1], 8 * sa) : sw[i]) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + 32 * u + lane;
            if (i < nw) dw[i] = v[u];
        }
    }
    const int t = n & 3;
    if (lane < t) dst[4 * nw + lane] = src[4 * nw + lane];
}

// n bytes by N lanes, as above.
template <int N>
__device__ __forceinline__ void lanes_copy(uint8_t *__restrict__ dst, const uint8_t *__restrict__ src, int n, int lane)
{
    const int h = min((int)((4 - (reinterpret_cast<uintptr_t>(dst) & 3)) & 3), n), nw = (n - h) >> 2;
    const uint32_t first = rd32u(src), last = rd32u(src + max(n - 4, 0));
    uint32_t *dw = reinterpret_cast<uint32_t *>(dst + h);
#pragma unroll 4
    for (int i = lane; i < nw; i += N) dw[i] = rd32u(src + h + 4 * i);
    if (lane < h) dst[lane] = (uint8_t)(first >> 8 * lane);
    const int t = n - h - 4 * nw;
    if (lane < t) dst[n - t + lane] = (uint8_t)(last >> 8 * (4 - t + lane));
}

// n <= 32 bytes, 4 per step, so that the cost follows n (most literal runs
// between matches are 0-4 bytes). Source and destination never overlap. May
// read up to 7 bytes past s + n (inputs carry tail room).
__device__ __forceinline__ void copy_short(uint8_t *__restrict__ d, const uint8_t *__restrict__ s, int n)
{
    for (int i = 0; i < n; i += 4) {
        const uint32_t w = rd32u(s + i);
        d[i] = (uint8_t)w;
        if (i + 1 < n) d[i + 1] = (uint8_t)(w >> 8);
        if (i + 2 < n) d[i + 2] = (uint8_t)(w >> 16);
        if (i + 3 < n) d[i + 3] = (uint8_t)(w >> 24);
    }
}

// Bytes of a length field's continuation: n/255 bytes of 255, then n%255.
__device__ __forceinline__ int len_bytes(int n) { return n / 255 + 1; }
__device__ __forceinline__ void put_len_serial(uint8_t *d, int n)
{
    for (; n >= 255; n -= 255) *d++ = 255;
    *d = (uint8_t)n;
}

// Record layout of a chunk: literal-only range [lo, hi) of the current
// record (its byte planes 1 and 2) and where the next record starts.
struct Skip {
    int lo, hi, next;
    bool on;
};
__device__ __forceinline__ void next_skip(Skip &k, const uint8_t *src, int L)
{
    while (k.on) {
        if (k.next + 4 > L) break;
        const int nb = (int)rd32u(src + k.next);
        if (nb < 4096 || nb > 4096 + 4 * 32768 || k.next + 4 + nb > L) break;
        const int S = (nb - 4096) / 4;
        k.lo = k.next + 4 + 4096 + S;
        k.hi = k.lo + 2 * S;
        k.next += 4 + nb;
        if (k.hi > k.lo) return;
    }
    k.on = false;
    k.lo = k.hi = L + 1;
}

// ------------------------------------------------------------------ encode
// Per warp, per super-window of kSW positions:
//   probe  -- 128 positions per step (4 per lane): hash, table lookup and
//             insert, verification against the stored 4-byte sequence;
//             the candidate offset per position goes to info[] (0: none);
//   walk   -- lane k walks positions [base+32k, base+32k+32) greedily
//             (take the match at the cursor, measure it, jump past it,
//             else step 1);
//   merge  -- lane k keeps its sequences that start at or after the end of
//             the last kept match of lanes < k: the kept matches never
//             overlap, so the parse stays valid LZ4 without any lane
//             waiting for another;
//   emit   -- every lane sizes its kept sequences, a warp scan places them,
//             every lane writes its own; literal runs longer than 32 bytes
//             are queued and copied by several lanes.
constexpr int kOvl = 8;
// super-window sizes: 768 positions when every chunk of the launch is
// resident at once (fewer windows per chunk), 512 otherwise (a smaller
// per-warp footprint, so more chunks share an SM)
constexpr int kWinSmall = 512, kWinLarge = 768;
constexpr int kMinHole = 256;  // smallest literal-only span left to the gather
// Hash table entry: position modulo 2^18 in the high bits, a 14-bit tag of
// the 4-byte sequence in the low bits. A tag hit is only a candidate: the
// walk measures the match from its first byte and drops it below 4 bytes.
constexpr uint32_t kPosMask = (1u << 18) - 1;
__device__ __forceinline__ uint32_t lz_tag(uint32_t v) { return (v * 0x85ebca77u) >> 18; }

// 8 bytes at any byte address as two little-endian words (three aligned
// loads). May read up to 11 bytes past p.
__device__ __forceinline__ void rd8u(const uint8_t *p, uint32_t (&v)[2])
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t sh = (uint32_t)(a & 3) * 8;
    const uint32_t x0 = w[0], x1 = w[1], x2 = w[2];
    v[0] = sh ? __funnelshift_r(x0, x1, sh) : x0;
    v[1] = sh ? __funnelshift_r(x1, x2, sh) : x1;
}

// exact match length from (p, cand), starting `known` bytes in (lane-local):
// the first 8 bytes on their own (most matches are 4-8 bytes long), then 16
// bytes per round trip to memory
__device__ __forceinline__ int match_len(const uint8_t *src, int p, int cand, int known, int matchlimit)
{
    int len = known;
    {
        uint32_t a[2], b[2];
        rd8u(src + p + len, a);
        rd8u(src + cand + len, b);
        const uint32_t x0 = a[0] ^ b[0], x1 = a[1] ^ b[1];
        const int k = x0 ? (__ffs(x0) - 1) >> 3 : x1 ? 4 + ((__ffs(x1) - 1) >> 3) : 8;
        len += k;
        if (k < 8) return len < matchlimit - p ? len : matchlimit - p;
    }
    while (p + len < matchlimit) {
        uint32_t a[4], b[4];
        rd16u(src + p + len, a);
        rd16u(src + cand + len, b);
        int k = 16;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
            const uint32_t x = a[j] ^ b[j];
            if (x) k = 4 * j + ((__ffs(x) - 1) >> 3);
        }
        len += k;
        if (k < 16) break;
    }
    return len < matchlimit - p ? len : matchlimit - p;
}

// match_len from byte 0, and how many of the (at most 4) bytes before p
// equal the bytes before cand (0 when cand < 4): the words before both
// positions are loaded with the first 8 bytes, so the count costs no
// extra round trip to memory.
__device__ __forceinline__ int match_len_back(const uint8_t *src, int p, int cand, int matchlimit, int &back)
{
    const uintptr_t pa = reinterpret_cast<uintptr_t>(src + p), ca = reinterpret_cast<uintptr_t>(src + cand);
    const uint32_t *pw = reinterpret_cast<const uint32_t *>(pa & ~(uintptr_t)3);
    const uint32_t *cw = reinterpret_cast<const uint32_t *>(ca & ~(uintptr_t)3);
    const uint32_t ps = (uint32_t)(pa & 3) * 8, cs = (uint32_t)(ca & 3) * 8;
    const bool before = cand >= 4;  // then p > cand >= 4 too: both words lie inside the chunk
    const uint32_t p0 = pw[0], p1 = pw[1], p2 = pw[2], pm = before ? pw[-1] : 0u;
    const uint32_t c0 = cw[0], c1 = cw[1], c2 = cw[2], cm = before ? cw[-1] : 0u;
    const uint32_t a0 = ps ? __funnelshift_r(p0, p1, ps) : p0, a1 = ps ? __funnelshift_r(p1, p2, ps) : p1;
    const uint32_t b0 = cs ? __funnelshift_r(c0, c1, cs) : c0, b1 = cs ? __funnelshift_r(c1, c2, cs) : c1;
    const uint32_t ab = ps ? __funnelshift_r(pm, p0, ps) : pm, bb = cs ? __funnelshift_r(cm, c0, cs) : cm;
    back = before ? __clz(ab ^ bb) >> 3 : 0;
    const uint32_t x0 = a0 ^ b0, x1 = a1 ^ b1;
    const int k = x0 ? (__ffs(x0) - 1) >> 3 : x1 ? 4 + ((__ffs(x1) - 1) >> 3) : 8;
    if (k < 8) return k < matchlimit - p ? k : matchlimit - p;
    return match_len(src, p, cand, 8, matchlimit);
}

// SEQ: the parse for the DEFLATE encoder instead of LZ4 bytes -- distances up
// to 32 KiB, and per kept sequence one 8-byte record (literal run, match
// length, distance; zl::seq_pack) at out + out_off[c]; the last record holds
// the tail literals. out_len[c] = record bytes, -1 past the capacity.
// Shared memory of one encoder warp for super-windows of SW positions.
// A lane's sequences, (start - base | back extension << 12 | offset << 16, match
// length), take the place of its positions' candidates: the i-th sequence ends
// at or after position 4 i + 4, where the walk's next read is. With OWN (effort
// 2, whose walks read the end of the lower lane's segment) they have their
// own.
template <int SW, bool OWN>
struct LzEncWarp {
    uint32_t table[1 << kHashLog];
    int4 longq[32];                   // (dst offset, src offset, n, -)
    uint16_t info[SW];                // candidate offset per position, 0: none
    uint2 own[OWN ? SW / 4 : 1];
    int nlong;
};

// With effort >= 1 a match [s, e) that starts before the literal position P is
// kept from P on when that part is still a match (>= 4 bytes) that may follow a
// literal run (P <= mflimit).
template <int kEffort>
__device__ __forceinline__ bool lz_survives(int s, int e, int P, int mflimit)
{
    return s >= P || (kEffort >= 1 && e - P >= kMinMatch && P <= mflimit);
}

// The parse of one chunk by one warp, window by window.
template <bool SEQ, int kEffort, int kSW>
struct LzParse {
    static constexpr int kSub = kSW / 32;  // positions per lane; a quarter as many sequences
    static constexpr bool kThorough = kEffort >= 2;
    static constexpr int kMaxOff = SEQ ? zl::kMaxDist : 65535;
    const uint8_t *src;
    int L, pos, anchor, miss, mflimit, matchlimit;
    int hlo, hhi;  // the literal-only planes last jumped over
    Skip sk;

    __device__ __forceinline__ void start(const uint8_t *s, int n, bool records, uint32_t *table)
    {
        for (int i = threadIdx.x & 31; i < (1 << kHashLog); i += 32) table[i] = kEmpty;
        __syncwarp();
        src = s;
        L = n;
        pos = anchor = miss = hlo = hhi = 0;
        sk.on = records;
        sk.next = 0;
        sk.lo = sk.hi = L + 1;
        if (sk.on) next_skip(sk, src, L);
        mflimit = L - kMfLimit;
        matchlimit = L - kLastLiterals;
    }

    // Up to the next window with candidates: its start, and the lane's ns
    // sequences (mine) from literal position myP on. False at the end.
    __device__ __forceinline__ bool next(uint32_t *table, uint16_t *info, uint2 *mine, int &base, int &ns, int &myP)
    {
        const int lane = threadIdx.x & 31;
        while (L >= kMfLimit + 1 && pos <= mflimit) {
            if (pos >= sk.lo) {  // literal-only planes: jump over them
                if (pos < sk.hi) pos = sk.hi;
                hlo = sk.lo;
                hhi = sk.hi;
                next_skip(sk, src, L);
                miss = 0;
                continue;
            }
            base = pos;
            int end = base + kSW;
            if (end > mflimit + 1) end = mflimit + 1;
            if (end > sk.lo) end = sk.lo;
            // ---- probe [base, end): the window's words are loaded up front
            // and the next window is prefetched into L1
            bool any_match = false;
            constexpr int kSteps = (kSW + 4 + 127) / 128;
            uint32_t wv[kSteps], wx[kSteps];
            // effort 2: the word before the window (for the distance 1-3
            // candidates of its first positions)
            uint32_t wprev = kThorough && (base & ~3) >= 4
                                 ? __ldg(reinterpret_cast<const uint32_t *>(src + (base & ~3) - 4))
                                 : 0u;
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const int wpos = (base & ~3) + 128 * k + 4 * lane;
                wv[k] = wpos + 4 <= L ? __ldg(reinterpret_cast<const uint32_t *>(src + wpos)) : 0u;
                wx[k] = lane == 31 && wpos + 8 <= L ? __ldg(reinterpret_cast<const uint32_t *>(src + wpos + 4)) : 0u;
            }
            if (lane < kSteps && (base & ~3) + kSW + 128 * lane < L)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(src + (base & ~3) + kSW + 128 * lane));
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const int wb = (base & ~3) + 128 * k;
                if (wb >= end) break;
                const int wpos = wb + 4 * lane;
                const uint32_t w0 = wv[k];
                uint32_t w1 = __shfl_down_sync(0xffffffffu, w0, 1);
                if (lane == 31) w1 = wx[k];
                // sx[3 + i]: the 4-byte sequence at wpos + i, i = -3..3
                // (i < 0 only with effort 2)
                uint32_t sx[7], h[4];
                bool valid[4];
                if (kThorough) {
                    uint32_t wp = __shfl_up_sync(0xffffffffu, w0, 1);
                    if (lane == 0) wp = wprev;
                    wprev = __shfl_sync(0xffffffffu, w0, 31);
#pragma unroll
                    for (int i = 0; i < 3; ++i) sx[i] = __funnelshift_r(wp, w0, 8 + 8 * i);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int p = wpos + j;
                    valid[j] = p >= base && p < end;
                    sx[3 + j] = j ? __funnelshift_r(w0, w1, 8 * j) : w0;
                    h[j] = lz_hash(sx[3 + j]);
                }
                const uint32_t *seq = sx + 3;
                uint32_t e[4], tag[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    e[j] = table[h[j]];
                    tag[j] = lz_tag(seq[j]);
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (valid[j]) table[h[j]] = (((uint32_t)(wpos + j) & kPosMask) << 14) | tag[j];
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int p = wpos + j;
                    const int off = (int)(((uint32_t)p - (e[j] >> 14)) & kPosMask);
                    int v = 0;
                    if (valid[j] && e[j] != kEmpty && (e[j] & 0x3fff) == tag[j] && off >= 1 && off <= kMaxOff && off <= p)
                        v = off;  // the walk verifies and measures chosen candidates
                    if (kThorough) {
                        // the table is read before this step's positions
                        // enter it, so a repeat at distance 1-3 (runs, short
                        // periods) is taken from the sequences directly
                        const int near = seq[j] == sx[2 + j] ? 1 : seq[j] == sx[1 + j] ? 2 : seq[j] == sx[j] ? 3 : 0;
                        if (near && p >= near) v = near;
                    }
                    if (valid[j]) info[p - base] = (uint16_t)v;
                    any_match |= v != 0;
                }
            }
            __syncwarp();
            if (!__any_sync(0xffffffffu, any_match)) {
                ++miss;
                pos = end + (miss > 2 ? (miss - 2) * 256 : 0);
                continue;
            }
            miss = 0;
            // ---- walk: lane-local greedy parse of [base + kSub*lane, +kSub)
            // (effort 2: entered kOvl positions early, at the end of the
            // lower lane's segment, so that it mostly lands on the serial
            // parse's path); a kept match also records how many bytes before
            // it equal the bytes before its source (at most 4), taken into
            // the match in the emission as far as the literal run allows
            // (effort >= 1: lz4.c's backward "catch up", lz4.c:586-587)
            ns = 0;
            int last_start = -1, last_end = -1;
            {
                const int w0p = base + kSub * lane;
                const int qe = min(w0p + kSub, end);
                const int qs = kThorough && lane ? w0p - kOvl : w0p;
                // the walk's positions that have a candidate (bit i: qs + i),
                // so that it jumps over literal positions
                constexpr int kNq = kThorough ? kSub + kOvl : kSub;
                uint32_t cm = 0;
                if (qe > qs) {
                    const uint4 *iv = reinterpret_cast<const uint4 *>(info + (qs - base));  // 16-byte aligned
#pragma unroll
                    for (int v = 0; v < kNq / 8; ++v) {
                        const uint4 a = iv[v];
                        const uint32_t iw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            cm |= (uint32_t)((iw[i] & 0xffffu) != 0) << (8 * v + 2 * i) |
                                  (uint32_t)((iw[i] >> 16) != 0) << (8 * v + 2 * i + 1);
                    }
                    if (qe - qs < kNq) cm &= (1u << (qe - qs)) - 1u;
                }
                int q = qs;
                while (q < qe) {
                    const uint32_t m = cm >> (q - qs);
                    if (!m) break;
                    q += __ffs(m) - 1;
                    const int off = info[q - base];
                    int ext = 0;
                    const int len = !off ? 0
                                    : kEffort >= 1 ? match_len_back(src, q, q - off, matchlimit, ext)
                                                   : match_len(src, q, q - off, 0, matchlimit);
                    if (len >= kMinMatch) {
                        if (q >= w0p) {
                            mine[ns++] = make_uint2((uint32_t)(q - base) | (uint32_t)ext << 12 | (uint32_t)off << 16,
                                                    (uint32_t)len);
                            last_start = q;
                            last_end = q + len;
                        }
                        q += len;
                    } else {
                        ++q;
                    }
                }
            }
            // ---- merge: P_k = end of the last kept match of lanes < k. With
            // effort >= 1 a match [s, e) that starts before the literal
            // position P is kept from P on when that part is still a match
            // (>= 4 bytes) that may follow a literal run (P <= mflimit).
            // Usually every lane keeps its last sequence, so P_k is the end
            // of the nearest lower lane's last match; where a match reaches
            // past a later lane's last start, the exact serial rule runs.
            const unsigned has = __ballot_sync(0xffffffffu, ns > 0);
            const unsigned lower = has & lanemask_lt_();
            myP = __shfl_sync(0xffffffffu, last_end, lower ? 31 - __clz(lower) : 0);
            if (!lower) myP = anchor;
            int P = has ? __shfl_sync(0xffffffffu, last_end, 31 - __clz(has)) : anchor;
            const unsigned bad = __ballot_sync(0xffffffffu, ns > 0 && !lz_survives<kEffort>(last_start, last_end, myP, mflimit));
            if (bad) {
                // lanes below the first failing one are exact; from there the
                // serial rule over the lanes that have sequences
                const int f = __ffs(bad) - 1;
                P = __shfl_sync(0xffffffffu, myP, f);
                for (unsigned rest = has & ~((1u << f) - 1u); rest; rest &= rest - 1u) {
                    const int k = __ffs(rest) - 1;
                    const int ls = __shfl_sync(0xffffffffu, last_start, k);
                    const int le = __shfl_sync(0xffffffffu, last_end, k);
                    if (lane == k) myP = P;
                    if (lz_survives<kEffort>(ls, le, P, mflimit)) P = le;
                }
            }
            anchor = P;
            pos = end > P ? end : P;
            return true;
        }
        return false;
    }
};

// Its output.
template <bool SEQ, int kEffort>
struct LzEmit {
    const uint8_t *src;
    uint8_t *dst;
    int L, cap, mflimit, op;
    // whether the chunk's one deferred copy (left to the gather) is taken
    bool deferred;
    int4 *hole;  // the chunk's, or nullptr

    __device__ __forceinline__ void start(const uint8_t *s, int n, uint8_t *d, int4 *h, bool records)
    {
        src = s;
        dst = d;
        L = n;
        cap = SEQ ? 8 * (L / 4 + 2) : L + L / 255 + 16;
        mflimit = L - kMfLimit;
        op = 0;
        hole = h;
        deferred = h == nullptr || !records;
        if (h && (threadIdx.x & 31) == 0) *h = make_int4(0, 0, 0, 0);  // written for every chunk
    }

    // A window's sequences; false past the capacity.
    __device__ __forceinline__ bool window(int base, int ns, int myP, const uint2 *mine, int hlo, int hhi, int4 *longq,
                                           int &nlong)
    {
        const int lane = threadIdx.x & 31;
        auto survives = [&](int s, int e, int P) { return lz_survives<kEffort>(s, e, P, mflimit); };
        // ---- emit: kept sequences are those starting at or after myP
        int lit_from = myP, bytes = 0, nkeep = 0;
        for (int i = 0; i < ns; ++i) {
            const uint2 w = mine[i];
            const int s0 = base + (int)(w.x & 0xfff), e0 = s0 + (int)w.y;
            if (!survives(s0, e0, lit_from)) continue;
            const int st = max(s0 - (int)((w.x >> 12) & 7), lit_from);
            const int l = st - lit_from, ml = e0 - st - kMinMatch;
            bytes += SEQ ? 8 : 1 + (l >= 15 ? len_bytes(l - 15) : 0) + l + 2 + (ml >= 15 ? len_bytes(ml - 15) : 0);
            lit_from = e0;
            ++nkeep;
        }
        int incl = bytes;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        if ((long long)op + total + 1 + kLastLiterals > cap) {
            return false;
        }
        if (lane == 0) nlong = 0;
        __syncwarp();
        if (SEQ) {
            int at = op + incl - bytes;
            lit_from = myP;
            for (int i = 0; i < ns; ++i) {
                const uint2 w = mine[i];
                const int s0 = base + (int)(w.x & 0xfff), e0 = s0 + (int)w.y;
                if (!survives(s0, e0, lit_from)) continue;
                const int st = max(s0 - (int)((w.x >> 12) & 7), lit_from);
                *reinterpret_cast<unsigned long long *>(dst + at) =
                    zl::seq_pack(st - lit_from, e0 - st, (int)(w.x >> 16));
                at += 8;
                lit_from = e0;
            }
        } else {
            int at = op + incl - bytes;
            lit_from = myP;
            for (int i = 0; i < ns; ++i) {
                const uint2 w = mine[i];
                const int s0 = base + (int)(w.x & 0xfff), e0 = s0 + (int)w.y;
                if (!survives(s0, e0, lit_from)) continue;
                const int st = max(s0 - (int)((w.x >> 12) & 7), lit_from);
                const int l = st - lit_from, ml = e0 - st - kMinMatch, off = (int)(w.x >> 16);
                uint8_t *d = dst + at;
                *d++ = (uint8_t)(((l >= 15 ? 15 : l) << 4) | (ml >= 15 ? 15 : ml));
                if (l >= 15) {
                    put_len_serial(d, l - 15);
                    d += len_bytes(l - 15);
                }
                if (l <= 32) {
                    copy_short(d, src + lit_from, l);
                } else {
                    const int slot = atomicAdd(&nlong, 1);
                    if (slot < 32) longq[slot] = make_int4((int)(d - dst), lit_from, l, 0);
                }
                d += l;
                d[0] = (uint8_t)off;
                d[1] = (uint8_t)(off >> 8);
                if (ml >= 15) put_len_serial(d + 2, ml - 15);
                at += 1 + (l >= 15 ? len_bytes(l - 15) : 0) + l + 2 + (ml >= 15 ? len_bytes(ml - 15) : 0);
                lit_from = e0;
            }
        }
        __syncwarp();
        const int nl = nlong;
        if (nl > 32) {  // cannot happen: a long run (> 32 bytes) only before a lane's first sequence
            return false;
        }
        // runs shorter than a hole: four at a time, 8 lanes each, so that
        // their loads overlap (a window has 3 to 4, of 33 to 100 bytes)
        for (int i = 0; i < nl; i += 4) {
            const int4 t = longq[min(i + (lane >> 3), 31)];
            if (i + (lane >> 3) < nl && t.z < kMinHole) lanes_copy<8>(dst + t.x, src + t.y, t.z, lane & 7);
        }
        for (int i = 0; i < nl; ++i) {
            const int4 t = longq[i];
            if (t.z < kMinHole) continue;
            // the planes inside this run go to the gather (once per
            // chunk): it copies them from the records into the stream
            const int a = max(t.y, hlo), b = min(t.y + t.z, hhi);
            if (!deferred && b - a >= kMinHole) {
                warp_copy(dst + t.x, src + t.y, a - t.y, lane);
                warp_copy(dst + t.x + (b - t.y), src + b, t.y + t.z - b, lane);
                if (lane == 0) *hole = make_int4(t.x + (a - t.y), a, b - a, 0);
                deferred = true;
            } else {
                warp_copy(dst + t.x, src + t.y, t.z, lane);
            }
        }
        __syncwarp();
        op += total;
        return true;
    }

    // The literals from anchor on; false past the capacity.
    __device__ __forceinline__ bool tail(int anchor, int hlo, int hhi)
    {
        const int lane = threadIdx.x & 31;
        if (SEQ) {
            if (op + 8 > cap) {
                return false;
            } else {
                if (lane == 0) *reinterpret_cast<unsigned long long *>(dst + op) = zl::seq_pack(L - anchor, 0, 0);
                op += 8;
            }
        } else {
            const int lit = L - anchor;
            const int need = 1 + (lit >= 15 ? len_bytes(lit - 15) : 0) + lit;
            if (op + need > cap) {
                return false;
            } else {
                if (lane == 0) {
                    dst[op] = (uint8_t)((lit >= 15 ? 15 : lit) << 4);
                    if (lit >= 15) put_len_serial(dst + op + 1, lit - 15);
                }
                op += 1 + (lit >= 15 ? len_bytes(lit - 15) : 0);
                const int a = max(anchor, hlo), b = min(L, hhi);
                if (!deferred && b - a >= kMinHole) {  // the planes to the gather, as above
                    warp_copy(dst + op, src + anchor, a - anchor, lane);
                    warp_copy(dst + op + (b - anchor), src + b, L - b, lane);
                    if (lane == 0) *hole = make_int4(op + (a - anchor), a, b - a, 0);
                    deferred = true;
                } else {
                    warp_copy(dst + op, src + anchor, lit, lane);
                }
                op += lit;
            }
        }
        return true;
    }
};

template <int kLzWarps, bool SEQ, int kEffort, int kSW>
__global__ void __launch_bounds__(kLzWarps * 32, 32 / kLzWarps)
lz4_encode_kernel(const uint8_t *__restrict__ in, const long long *in_off, const int *in_len, int nchunks,
                  uint8_t *__restrict__ out, const long long *out_off, int *out_len, int records, int4 *hole)
{
    using Parse = LzParse<SEQ, kEffort, kSW>;
    using LzEncWarp = cz::LzEncWarp<kSW, Parse::kThorough>;
    // up to 8 warps in static shared memory; 16 in dynamic
    extern __shared__ __align__(16) unsigned char lz_enc_smem[];
    __shared__ LzEncWarp lz_enc_static[kLzWarps <= 8 ? kLzWarps : 1];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    LzEncWarp &ws = (kLzWarps <= 8 ? lz_enc_static : reinterpret_cast<LzEncWarp *>(lz_enc_smem))[wib];
    uint2 *mine = (Parse::kThorough ? ws.own : reinterpret_cast<uint2 *>(ws.info)) + Parse::kSub / 4 * lane;
    const int gw = blockIdx.x * kLzWarps + wib, nw = gridDim.x * kLzWarps;

    for (int c = gw; c < nchunks; c += nw) {
        const uint8_t *src = in + in_off[c];
        const int L = in_len[c];
        Parse p;
        LzEmit<SEQ, kEffort> e;
        p.start(src, L, records != 0, ws.table);
        e.start(src, L, out + out_off[c], hole ? hole + c : nullptr, records != 0);
        bool ok = true;
        int base, ns, myP;
        while (ok && p.next(ws.table, ws.info, mine, base, ns, myP))
            ok = e.window(base, ns, myP, mine, p.hlo, p.hhi, ws.longq, ws.nlong);
        ok = ok && e.tail(p.anchor, p.hlo, p.hhi);
        if (lane == 0) out_len[c] = ok ? e.op : -1;
        __syncwarp();
    }
}

// Two warps per chunk, for few chunks: one parses, the other writes what the
// window before gave. A chunk is one serial chain of windows (a window's start
// and its table depend on the window before; about 6 k cycles of parse and
// 5 k of output each, nearly all latency), so this takes it through nearly
// twice as fast while there are SMs for the second warps. Same bytes.
template <int SW>
struct LzPairShared {
    uint32_t table[1 << kHashLog];
    int4 longq[32];
    uint16_t info[SW];
    uint2 seq[2][SW / 4];  // two windows in flight
    int2 lane[2][32];      // ns, myP
    int4 win[2];           // base (-1: the end, with the anchor), anchor, hlo, hhi
    int nlong;
};
// Named barriers, one per buffer b: 1 + b full, 3 + b empty. Immediate ids, so
// that a CTA holds 5 of the SM's barriers and not 16.
template <int ID>
__device__ __forceinline__ void pair_wait(int b)
{
    if (b) asm volatile("bar.sync %0, 64;" ::"n"(ID + 1) : "memory");
    else asm volatile("bar.sync %0, 64;" ::"n"(ID) : "memory");
}
template <int ID>
__device__ __forceinline__ void pair_signal(int b)
{
    if (b) asm volatile("bar.arrive %0, 64;" ::"n"(ID + 1) : "memory");
    else asm volatile("bar.arrive %0, 64;" ::"n"(ID) : "memory");
}
constexpr int kPairFull = 1, kPairEmpty = 3;

template <bool SEQ, int kEffort, int kSW>
__global__ void __launch_bounds__(64)
lz4_encode_pair_kernel(const uint8_t *__restrict__ in, const long long *in_off, const int *in_len, int nchunks,
                       uint8_t *__restrict__ out, const long long *out_off, int *out_len, int records, int4 *hole)
{
    using Parse = LzParse<SEQ, kEffort, kSW>;
    __shared__ LzPairShared<kSW> ps;
    const int lane = threadIdx.x & 31;
    int buf = 0;
    if (threadIdx.x < 32) {
        for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
            Parse p;
            p.start(in + in_off[c], in_len[c], records != 0, ps.table);
            for (bool more = true; more; buf ^= 1) {
                pair_wait<kPairEmpty>(buf);
                int base, ns, myP;
                more = p.next(ps.table, ps.info, ps.seq[buf] + Parse::kSub / 4 * lane, base, ns, myP);
                if (more) ps.lane[buf][lane] = make_int2(ns, myP);
                if (lane == 0) ps.win[buf] = make_int4(more ? base : -1, p.anchor, p.hlo, p.hhi);
                pair_signal<kPairFull>(buf);
            }
        }
        // the buffers' last signals
        pair_wait<kPairEmpty>(buf);
        pair_wait<kPairEmpty>(buf ^ 1);
    } else {
        pair_signal<kPairEmpty>(0);
        pair_signal<kPairEmpty>(1);
        for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
            LzEmit<SEQ, kEffort> e;
            e.start(in + in_off[c], in_len[c], out + out_off[c], hole ? hole + c : nullptr, records != 0);
            bool ok = true;  // past the capacity the rest of the chunk's windows are passed over
            for (bool more = true; more; buf ^= 1) {
                pair_wait<kPairFull>(buf);
                const int4 w = ps.win[buf];
                more = w.x >= 0;
                if (more && ok) {
                    const int2 l = ps.lane[buf][lane];
                    ok = e.window(w.x, l.x, l.y, ps.seq[buf] + Parse::kSub / 4 * lane, w.z, w.w, ps.longq, ps.nlong);
                } else if (ok) {
                    ok = e.tail(w.y, w.z, w.w);
                }
                __syncwarp();
                pair_signal<kPairEmpty>(buf);
            }
            if (lane == 0) out_len[c] = ok ? e.op : -1;
        }
    }
}

// ------------------------------------------------------------------ decode
// n bytes from s to d by the CTA: bytes until d is 16-byte aligned, then
// 16-byte stores (each built from five 4-byte loads with funnel shifts), then
// the tail. Wide stores matter when the destination is host memory written
// over the CPU-GPU link. Reads up to 4 bytes past s + n.
__device__ __forceinline__ void cta_copy(uint8_t *__restrict__ d, const uint8_t *__restrict__ s, int n)
{
    if (n <= 0) return;
    int h = (int)((16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15);
    if (h > n) h = n;
    if ((int)threadIdx.x < h) d[threadIdx.x] = s[threadIdx.x];
    const uint8_t *s2 = s + h;
    uint4 *dw = reinterpret_cast<uint4 *>(d + h);
    const int m = n - h, nwd = m >> 4;
    const uint32_t sa = (uint32_t)(reinterpret_cast<uintptr_t>(s2) & 3);
    const uint32_t *sw = reinterpret_cast<const uint32_t *>(s2 - sa);
    for (int i = threadIdx.x; i < nwd; i += blockDim.x) {
        const uint32_t *q = sw + 4 * i;
        const uint32_t a0 = q[0], a1 = q[1], a2 = q[2], a3 = q[3], a4 = sa ? q[4] : 0u;
        uint4 v;
        if (sa) {
            v.x = __funnelshift_r(a0, a1, 8 * sa);
            v.y = __funnelshift_r(a1, a2, 8 * sa);
            v.z = __funnelshift_r(a2, a3, 8 * sa);
            v.w = __funnelshift_r(a3, a4, 8 * sa);
        } else {
            v = make_uint4(a0, a1, a2, a3);
        }
        dw[i] = v;
    }
    const int t = m & 15;
    if ((int)threadIdx.x < t) d[h + 16 * nwd + threadIdx.x] = s2[16 * nwd + threadIdx.x];
}

// Input bytes of chunk c, -1 for a length that cannot be.
__device__ __forceinline__ int chunk_len(const long long *in_off, const int *in_len, int c)
{
    if (in_len) return in_len[c];
    const long long n = in_off[c + 1] - in_off[c];
    return n < 0 || n > 0x7fffffffLL ? -1 : (int)n;
}

// One CTA per chunk, for few chunks. The chunk is one serial chain of sequences, each of a few
// bytes; what bounds a decoder is that chain and, with many chunks, issue.
// Both want many sequences per step, so a step takes kDecIn input bytes:
//   * every warp decodes the tokens at all 128 positions of its window as if
//     a sequence started there (4 per lane) and makes jump tables by pointer
//     doubling in shared memory: T_b, 2^b steps along the next-token chain,
//     positions past the window absorbing. T_6 is then the window's exit for
//     every entry, so the chain through the step's windows costs one lookup
//     each, and lane k finds the window's k-th sequence in six;
//   * thread t takes the step's t-th sequence; scans give output positions,
//     and the reference's acceptance tests run per sequence, the first that
//     does not pass ends the step;
//   * the output is made in a ring in shared memory, a word per thread and
//     turn (its sequence by binary search over the output positions):
//     literals and match bytes whose source lies before the step are written
//     at once, other match bytes leave their distance, and are then chased
//     along the distances to a written byte, every hop adding the distance
//     that the byte met holds by then, so that chains of copies of copies
//     shorten for all at once (pointer jumping) without a barrier per round.
// Sequences with length fields of more than kFastExt bytes, or too long for
// the ring, are decoded serially, their copies by the whole CTA.
// A step of 1 KB of input (about 180 sequences) takes 10 k cycles on an SM of
// its own; one-record chunks on an idle GPU 0.18 ms instead of 0.61 with one
// warp each (64 chunks of a 128^3 field), 15-record chunks 2.33 instead of
// 9.0 ms (35 chunks of a 256^3 field).
constexpr int kDecWarps = 8, kDecThreads = 32 * kDecWarps;
constexpr int kWin = 128, kLevels = 7, kFastExt = 8;
constexpr int kDecIn = kWin * kDecWarps;     // input positions per step
constexpr int kDecStage = kDecIn + 64;       // input bytes held in shared memory
constexpr int kMaxSeqWin = (kWin + 2) / 3;   // a sequence takes at least 3 input bytes
// A step adds at most kStage bytes, so at least kRing - kStage - 4 bytes of
// history stay readable while it is written. Of the match sources in
// block-record chunks 90% lie within 3 KB and 99% within 12 KB, but a single
// source in global memory costs its whole step an L2 round trip: with 16 KB
// instead of 32 a launch of 2048 chunks took 0.627 ms instead of 0.514.
constexpr int kRing = 32768, kMask = kRing - 1, kStage = 4096;
constexpr uint32_t kEnd = 0xffffu;  // next position of a sequence that ends the chain (last, or serial)

// Sum of the length continuation bytes from ip while they are 255 and
// ip < lim; leaves ip after the last byte read. Called by whole warps.
__device__ __forceinline__ long long get_len(const uint8_t *src, int &ip, int lim, int lane)
{
    long long sum = 0;
    while (ip < lim) {
        const int b = ip + lane < lim ? (int)__ldg(src + ip + lane) : -1;
        const unsigned stop = __ballot_sync(0xffffffffu, b != 255);
        const int k = stop ? __ffs(stop) - 1 : 32;  // bytes of 255 first
        sum += 255ll * k;
        ip += k;
        if (k < 32) {
            const int last = __shfl_sync(0xffffffffu, b, k);
            if (last >= 0) {
                sum += last;
                ++ip;
            }
            break;
        }
    }
    return sum;
}

// Byte k of a match at output ms comes from ms - off + (k mod off): the
// byte-serial copy repeats the first `off` bytes when off < length.
__device__ __forceinline__ int msrc(int k, int off, int ml) { return off >= ml ? k : k % off; }

// Byte planes 1 and 2 of a record chunk that the decoder left in its input
// (a literal run it did not copy): output [out, out + len) is input
// [in, in + len); len 0: none.
struct LzHole {
    int out = 0, len = 0, in = 0;
};

// Output byte x from global memory: from the input inside the hole, else
// from the output (via L2).
__device__ __forceinline__ uint8_t old_byte(const uint8_t *src, const uint8_t *dst, const LzHole &h, int x)
{
    return (unsigned)(x - h.out) < (unsigned)h.len ? __ldg(src + h.in + (x - h.out)) : __ldcg(dst + x);
}

// A decoded token.
struct LzSeq {
    int lit_at, lit, ml, next;  // literals' input position and count, match length, position after the sequence
    bool term, slow;            // ends the input; length field too long for the parallel parse
};

struct LzDecShared {
    uint8_t ring[kRing + 16];              // recent output (16 bytes of slack)
    uint16_t dist[kStage + 8];             // per output byte of the step (from its first word): distance to its source in the step, or 0
    uint16_t jump[kDecWarps][kLevels][kWin];  // T_b, positions relative to the step
    int4 seq[kDecThreads + 1];             // per sequence: output start, literals' end, input - output position of the literals, distance
    uint32_t in[kDecStage / 4 + 1];        // the step's input
    uint16_t first[kDecThreads];           // output start per sequence
    uint16_t slot[kDecWarps][kMaxSeqWin + 1];  // positions of each window's sequences
    int count[kDecWarps], bytes[kDecWarps];    // sequences and output bytes per warp
    int stop[kDecWarps], epos[kDecWarps], stop_at[kDecWarps], stop_pos[kDecWarps];  // first sequence not taken
    int exit;                              // the chain's position after the step
};

__global__ void __launch_bounds__(kDecThreads, 3)
lz4_decode_wide_kernel(const uint8_t *__restrict__ in, const long long *in_off, const int *in_len, int nchunks,
                  uint8_t *__restrict__ out, const long long *out_off, const int *out_cap, int *out_len,
                  int4 *hole, long long cap)
{
    extern __shared__ __align__(16) unsigned char lz_dec_smem[];
    LzDecShared &s = *reinterpret_cast<LzDecShared *>(lz_dec_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t *ring = s.ring;
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint8_t *src = in + in_off[c];
        const int iend = chunk_len(in_off, in_len, c);
        uint8_t *dst = out + (out_off ? out_off[c] : c * cap);
        const int oend = out_off ? out_cap[c] : (int)cap;
        int s0 = 0, op = 0, err = 0, ring_lo = 0;  // output before ring_lo is not in the ring
        bool done = false;
        LzHole hl;
        if (hole && tid == 0) hole[c] = make_int4(0, 0, 0, 0);  // written for every chunk
        __syncthreads();  // the previous chunk has left shared memory
        // a literal run of n bytes from input i to output o, except the
        // record's byte planes 1 and 2 when it covers them whole (hole
        // given, record chunks: the record's byte count is output bytes 0-3)
        auto lit_run = [&](int o, int i, int n) {
            int a = 0, b = 0;
            if (hole && hl.len == 0 && o >= 4) {
                const int nb = (int)__ldcg(dst) | (int)__ldcg(dst + 1) << 8 | (int)__ldcg(dst + 2) << 16 |
                               (int)__ldcg(dst + 3) << 24;
                if (nb >= 4096 && nb <= 4096 + 4 * 32768 && ((nb - 4096) & 3) == 0) {
                    const int S = (nb - 4096) >> 2;
                    a = 4 + 4096 + S;
                    b = a + 2 * S;
                    if (!(o <= a && o + n >= b && b - a >= kMinHole)) a = b = 0;
                }
            }
            if (b > a) {
                cta_copy(dst + o, src + i, a - o);
                cta_copy(dst + b, src + i + (b - o), o + n - b);
                hl.out = a;
                hl.len = b - a;
                hl.in = i + (a - o);
                if (tid == 0) hole[c] = make_int4(hl.out, hl.in, hl.len, 0);
            } else {
                cta_copy(dst + o, src + i, n);
            }
        };
        if (iend <= 0) {
            if (tid == 0) out_len[c] = 0;  // lz4.c:836: error exit at position 0
            continue;
        }
        // word i of the input around position p (whole aligned words; none
        // that lies past the input)
        auto in_word = [&](int p, int i) -> uint32_t {
            const uint8_t *a = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(src + p) & ~(uintptr_t)3) +
                               4 * i;
            return a < src + iend ? __ldg(reinterpret_cast<const uint32_t *>(a)) : 0u;
        };
        int ahead_at = -1;  // position the words loaded ahead belong to
        uint32_t ahead = 0, ahead2 = 0;
        constexpr int kExtra = kDecStage / 4 + 1 - kDecThreads;  // words beyond one per thread
        while (!done && !err) {
            // ---- the step's input; positions count from the aligned base
            const int base = s0 - (int)(reinterpret_cast<uintptr_t>(src + s0) & 3);
            if (ahead_at != s0) {
                ahead = in_word(s0, tid);
                ahead2 = tid < kExtra ? in_word(s0, kDecThreads + tid) : 0u;
            }
            s.in[tid] = ahead;
            if (tid < kExtra) s.in[kDecThreads + tid] = ahead2;
            __syncthreads();
            const uint8_t *ib = reinterpret_cast<const uint8_t *>(s.in);
            auto byte_at = [&](int p) -> int { return p - base < kDecStage ? (int)ib[p - base] : (int)__ldg(src + p); };
            // the token at p (< iend) as a sequence (lz4.c:846-882)
            auto decode = [&](int p, int tok) {
                LzSeq q;
                q.lit = tok >> 4;
                q.ml = tok & 15;
                q.lit_at = p + 1;
                q.next = 0;
                q.slow = q.term = false;
                if (q.lit == 15 && q.lit_at < iend) {
                    int e = byte_at(q.lit_at++);
                    q.lit += e;
                    if (e == 255) {  // rare
                        int k = 1;
                        for (; k < kFastExt && e == 255 && q.lit_at < iend; ++k) {
                            e = byte_at(q.lit_at++);
                            q.lit += e;
                        }
                        q.slow = e == 255 && q.lit_at < iend;
                    }
                }
                if (!q.slow && q.lit > iend - q.lit_at - (2 + 1 + kLastLiterals)) q.term = true;  // lz4.c:851
                if (!q.slow && !q.term) {
                    q.next = q.lit_at + q.lit + 2;
                    const int lim = iend - (kLastLiterals + 1);
                    if (q.ml == 15 && q.next < lim) {
                        int e = byte_at(q.next++);
                        q.ml += e;
                        if (e == 255) {
                            int k = 1;
                            for (; k < kFastExt && e == 255 && q.next < lim; ++k) {
                                e = byte_at(q.next++);
                                q.ml += e;
                            }
                            q.slow = e == 255 && q.next < lim;
                        }
                    }
                }
                q.ml += kMinMatch;
                return q;
            };
            // ---- jump tables of this warp's window
            const int w0 = warp * kWin;  // relative to base
            uint16_t(*T)[kWin] = s.jump[warp];
            uint32_t t0[4];
            {
                const uint32_t word = s.in[(w0 >> 2) + lane];
                const int p0 = base + w0 + 4 * lane;
                unsigned ext = 0;  // candidates with a length continuation
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int p = p0 + j, tok = (int)((word >> (8 * j)) & 0xff), lit = tok >> 4;
                    const bool in = p >= s0 && p < iend;
                    const bool plain = lit != 15 && (tok & 15) != 15;
                    if (in && !plain) ext |= 1u << j;
                    t0[j] = in && plain && lit <= iend - p - (1 + 2 + 1 + kLastLiterals) ? (uint32_t)(p - base + 3 + lit)
                                                                                        : kEnd;
                }
                while (ext) {
                    const int j = __ffs(ext) - 1;
                    ext &= ext - 1;
                    const LzSeq q = decode(p0 + j, (int)((word >> (8 * j)) & 0xff));
                    const uint32_t v = q.slow || q.term ? kEnd : (uint32_t)(q.next - base);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (i == j) t0[i] = v;
                }
                reinterpret_cast<uint2 *>(T[0])[lane] = make_uint2(t0[0] | t0[1] << 16, t0[2] | t0[3] << 16);
            }
            __syncwarp();
#pragma unroll
            for (int b = 1; b < kLevels; ++b) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (t0[j] - (uint32_t)w0 < (uint32_t)kWin) t0[j] = T[b - 1][t0[j] - w0];
                reinterpret_cast<uint2 *>(T[b])[lane] = make_uint2(t0[0] | t0[1] << 16, t0[2] | t0[3] << 16);
                __syncwarp();
            }
            __syncthreads();
            // ---- the chain through the windows, then this window's sequences
            uint32_t e = (uint32_t)(s0 - base);
            for (int w = 0; w < warp; ++w)
                if (e - (uint32_t)(w * kWin) < (uint32_t)kWin) e = s.jump[w][kLevels - 1][e - w * kWin];
            int cnt = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = lane + 32 * h;
                uint32_t pos = e;
#pragma unroll
                for (int b = 0; b < kLevels - 1; ++b)
                    if ((k >> b) & 1)
                        if (pos - (uint32_t)w0 < (uint32_t)kWin) pos = T[b][pos - w0];
                const bool member = k < kMaxSeqWin && pos - (uint32_t)w0 < (uint32_t)kWin;
                if (member) s.slot[warp][k] = (uint16_t)pos;
                cnt += __popc(__ballot_sync(0xffffffffu, member));
            }
            if (lane == 0) s.count[warp] = cnt;
            if (warp == kDecWarps - 1 && lane == 0)
                s.exit = (int)(e - (uint32_t)w0 < (uint32_t)kWin ? T[kLevels - 1][e - w0] : e);
            __syncthreads();
            // ---- thread t takes sequence t
            int nseq = 0, mw = 0, mk = tid, over = -1;  // over: position of sequence kDecThreads, if there is one
#pragma unroll
            for (int w = 0; w < kDecWarps; ++w) {
                const int n = s.count[w];
                if (tid >= nseq) {
                    mw = w;
                    mk = tid - nseq;
                }
                if (kDecThreads - nseq >= 0 && kDecThreads - nseq < n) over = s.slot[w][kDecThreads - nseq];
                nseq += n;
            }
            const int nthis = min(nseq, kDecThreads);
            const bool member = tid < nthis;
            const int after = over >= 0 ? over : s.exit;  // kEnd: the last sequence is terminal or slow
            // the next step's input, loaded ahead
            ahead_at = after != (int)kEnd ? base + after : -1;
            if (ahead_at >= 0) {
                ahead = in_word(ahead_at, tid);
                ahead2 = tid < kExtra ? in_word(ahead_at, kDecThreads + tid) : 0u;
            }
            int pos = 0, off = 0, stop = 0, epos = 0;  // stop 1: end of input, 2: malformed, 3: decode serially, 4: no room
            LzSeq q;
            q.lit_at = q.lit = q.ml = q.next = 0;
            q.term = q.slow = false;
            if (member) {
                pos = s.slot[mw][mk];
                q = decode(base + pos, (int)ib[pos]);
                if (!q.term && !q.slow) off = byte_at(q.lit_at + q.lit) | byte_at(q.lit_at + q.lit + 1) << 8;
            }
            const int len = member && !q.slow ? q.lit + (q.term ? 0 : q.ml) : 0;
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) s.bytes[warp] = incl;
            __syncthreads();
            int before = 0, total = 0;
#pragma unroll
            for (int w = 0; w < kDecWarps; ++w) {
                const int n = s.bytes[w];
                before += w < warp ? n : 0;
                total += n;
            }
            incl += before;  // output bytes of the step up to this sequence's end
            const int at = incl - len, opl = op + at, ms = opl + q.lit;
            // ---- acceptance tests (lz4.c:851-858, :868, :888-890)
            if (member) {
                if (q.slow) {
                    stop = 3;
                } else if (incl > kStage) {
                    stop = 4;
                } else if (q.term || q.lit > oend - opl - kMfLimit) {
                    if (q.lit > oend - opl || q.lit != iend - q.lit_at) {
                        stop = 2;
                        epos = q.lit_at;
                    } else {
                        stop = 1;
                    }
                } else if (off == 0 || off > ms) {
                    stop = 2;
                    epos = q.lit_at + q.lit + 2;
                } else if (q.ml > oend - ms - kLastLiterals) {
                    stop = 2;
                    epos = q.next;
                }
            }
            {
                const unsigned sb = __ballot_sync(0xffffffffu, stop != 0);
                const int k = sb ? __ffs(sb) - 1 : 0;
                const int why = __shfl_sync(0xffffffffu, stop, k), ep = __shfl_sync(0xffffffffu, epos, k);
                const int sat = __shfl_sync(0xffffffffu, at + (stop == 1 ? q.lit : 0), k),
                          sp = __shfl_sync(0xffffffffu, pos, k);
                if (lane == 0) {
                    s.stop[warp] = sb ? (32 * warp + k) << 3 | why : 0x7fffffff;
                    s.epos[warp] = ep;
                    s.stop_at[warp] = sat;
                    s.stop_pos[warp] = sp;
                }
            }
            s.first[tid] = (uint16_t)(member ? min(at, kStage) : kStage);
            s.seq[tid] = make_int4(at, at + q.lit, q.lit_at - at, off);
            __syncthreads();
            // the output ends where the first sequence that is not taken
            // starts (or ends, when it is the input's last literals)
            int ks = 0x7fffffff, kepos = 0, nout = total, kpos = 0;
#pragma unroll
            for (int w = kDecWarps - 1; w >= 0; --w)
                if (s.stop[w] < ks) {
                    ks = s.stop[w];
                    kepos = s.epos[w];
                    nout = s.stop_at[w];
                    kpos = s.stop_pos[w];
                }
            const int kstop = ks == 0x7fffffff ? 0 : ks & 7, kthread = ks >> 3;
            // ---- the output words: literals, history, distances
            const int lead = op & 3;  // bytes of the first word written by earlier steps
            const int lo = max(ring_lo, op + kStage + 4 - kRing);  // not overwritten by this step
            const int ngroup = nout > 0 ? (lead + nout + 3) >> 2 : 0;
            for (int g = tid; g < ngroup; g += kDecThreads) {
                const int i0 = 4 * g - lead;  // step-relative position of the word's first byte
                // the sequence that holds byte max(i0, 0): its warp, then within it
                int k = 0, sum = 0;
#pragma unroll
                for (int w = 0; w < kDecWarps - 1; ++w) {
                    sum += s.bytes[w];
                    if (sum <= i0) k = 32 * (w + 1);
                }
#pragma unroll
                for (int step = 16; step; step >>= 1)
                    if ((int)s.first[k + step] <= i0) k += step;
                const int4 A = s.seq[k], B = s.seq[k + 1];
                const int nextb = k + 1 < nthis ? B.x : 0x7fffffff;
                uint32_t word = i0 < 0 ? *reinterpret_cast<const uint32_t *>(ring + ((op + i0) & kMask)) : 0u;
                uint32_t d[4], v[4];
                unsigned far = 0;  // bytes that lie in global memory (rare)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = i0 + j;
                    const bool second = i >= nextb;
                    const int lend = second ? B.y : A.y, lsrc = second ? B.z : A.z, f = second ? B.w : A.w;
                    const bool lit = i < lend, live = i >= 0 && i < nout, here = live && (lit || f > i);
                    const int x = op + i - f, p = i + lsrc - base;
                    d[j] = live && !here ? (uint32_t)f : 0u;
                    const bool near = lit ? p < kDecStage : x >= lo;
                    v[j] = 0;
                    if (here && near) v[j] = lit ? ib[p] : ring[x & kMask];
                    if (here && !near) far |= 1u << j;
                    if (here) word &= ~(0xffu << (8 * j));
                }
                while (far) {
                    const int j = __ffs(far) - 1, i = i0 + j;
                    far &= far - 1;
                    const bool second = i >= nextb;
                    const int lend = second ? B.y : A.y, lsrc = second ? B.z : A.z, f = second ? B.w : A.w;
                    const uint32_t b = i < lend ? __ldg(src + i + lsrc) : old_byte(src, dst, hl, op + i - f);
                    word |= b << (8 * j);
                }
                word |= v[0] | v[1] << 8 | v[2] << 16 | v[3] << 24;
                *reinterpret_cast<uint32_t *>(ring + ((op + i0) & kMask)) = word;
                reinterpret_cast<uint2 *>(s.dist)[g] = make_uint2(d[0] | d[1] << 16, d[2] | d[3] << 16);
            }
            __syncthreads();
            // ---- the bytes that copy bytes of this step: along the distances to
            // a written byte (a byte's own distance only ever grows towards it)
            for (int g = tid; g < ngroup; g += kDecThreads) {
                const uint2 dw = reinterpret_cast<const uint2 *>(s.dist)[g];
                if ((dw.x | dw.y) == 0u) continue;
                volatile uint16_t *dist = s.dist;
                const int i = 4 * g;  // counted from the first word
                const uint32_t e0 = dw.x & 0xffffu, e1 = dw.x >> 16, e2 = dw.y & 0xffffu, e3 = dw.y >> 16;
                // the four bytes hop together; a byte that has arrived meets 0
                // (one without a distance meets itself)
                int x0 = i - (int)e0, x1 = i + 1 - (int)e1, x2 = i + 2 - (int)e2, x3 = i + 3 - (int)e3;
                for (;;) {
                    const uint32_t a0 = dist[x0], a1 = dist[x1], a2 = dist[x2], a3 = dist[x3];
                    if (!(a0 | a1 | a2 | a3)) break;
                    x0 -= (int)a0;
                    x1 -= (int)a1;
                    x2 -= (int)a2;
                    x3 -= (int)a3;
                    if (a0) dist[i] = (uint16_t)(i - x0);
                    if (a1) dist[i + 1] = (uint16_t)(i + 1 - x1);
                    if (a2) dist[i + 2] = (uint16_t)(i + 2 - x2);
                    if (a3) dist[i + 3] = (uint16_t)(i + 3 - x3);
                }
                const int o = op - lead;
                const uint8_t v0 = ring[(o + x0) & kMask], v1 = ring[(o + x1) & kMask], v2 = ring[(o + x2) & kMask],
                              v3 = ring[(o + x3) & kMask];
                if (e0) ring[(o + i) & kMask] = v0;
                if (e1) ring[(o + i + 1) & kMask] = v1;
                if (e2) ring[(o + i + 2) & kMask] = v2;
                if (e3) ring[(o + i + 3) & kMask] = v3;
            }
            __syncthreads();
            {
                const int r = op & kMask, n1 = min(nout, kRing - r);
                flush(dst + op, ring, r, n1, tid, kDecThreads);
                if (nout > n1) flush(dst + op + n1, ring, 0, nout - n1, tid, kDecThreads);
            }
            // ---- advance
            op += nout;
            if (kstop == 0) {
                s0 = base + after;
            } else if (kstop == 1) {
                done = true;
            } else if (kstop == 2) {
                err = kepos;
            } else if (kstop == 4 && kthread > 0) {
                s0 = base + kpos;
            } else {
                // a sequence with long length fields or a long output, decoded serially
                int ip = base + kpos;
                __syncthreads();  // the flushed output
                const int token = __ldg(src + ip);
                ++ip;
                long long ll = token >> 4;
                if (ll == 15) ll += get_len(src, ip, iend, lane);
                if (ll > (long long)(oend - op - kMfLimit) || ll > (long long)(iend - ip - (2 + 1 + kLastLiterals))) {
                    if (ll > (long long)(oend - op) || ll != (long long)(iend - ip)) {
                        err = ip;
                    } else {
                        lit_run(op, ip, (int)ll);
                        op += (int)ll;
                        done = true;
                    }
                } else {
                    lit_run(op, ip, (int)ll);
                    op += (int)ll;
                    ip += (int)ll;
                    const int o = (int)__ldg(src + ip) | ((int)__ldg(src + ip + 1) << 8);
                    ip += 2;
                    if (o == 0 || o > op) {
                        err = ip;
                    } else {
                        long long m = token & 15;
                        if (m == 15) m += get_len(src, ip, iend - (kLastLiterals + 1), lane);
                        m += kMinMatch;
                        if (m > (long long)(oend - op - kLastLiterals)) {
                            err = ip;
                        } else {
                            __syncthreads();
                            for (int k = tid; k < (int)m; k += kDecThreads)
                                dst[op + k] = old_byte(src, dst, hl, op - o + msrc(k, o, (int)m));
                            op += (int)m;
                            s0 = ip;
                            ring_lo = op;  // written around the ring
                        }
                    }
                }
            }
            __syncthreads();
        }
        if (tid == 0) out_len[c] = err ? -err : op;
    }
}

// One warp per chunk, for many chunks. The decoder reads a window of kWin input bytes starting
// at the current sequence. Every lane decodes the token at 4 candidate
// positions as if a sequence started there (literal length, offset, match
// length, position of the next token); only the candidates reachable from
// the window's first position are real sequences. Jump tables T_b (2^b
// steps along the next-token chain, built by pointer doubling in shared
// memory) let lane k find the k-th sequence directly. Candidates whose
// length fields run longer than kFastExt continuation bytes are flagged
// and decoded serially when the chain reaches them.
constexpr int kExit = kWin;
// Output ring per warp: the last kRing1 bytes of output. A window adds at
// most kStage1 bytes, so at least kRing1 - kStage1 bytes of history stay
// readable while it is written (about 99% of match sources in block-record
// chunks lie within 3 KB).
constexpr int kRing1 = 4096, kMask1 = kRing1 - 1, kStage1 = 1024;
constexpr int kTermIn = 1 << 16, kSlow = 1 << 17;  // flags above the 16-bit offset

// Continuation bytes like get_len, at most kFastExt of them: false if the
// field is longer (the caller then decodes the sequence serially).
__device__ __forceinline__ bool get_len_fast(const uint8_t *src, int &ip, int lim, int &sum)
{
#pragma unroll 1
    for (int k = 0; k < kFastExt; ++k) {
        if (ip >= lim) return true;
        const int s = __ldg(src + ip++);
        sum += s;
        if (s != 255) return true;
    }
    return ip >= lim;
}

// n <= 8 bytes from read-only input into the ring at output position o;
// all loads before the stores.
__device__ __forceinline__ void copy_lit(uint8_t *ring, int o, const uint8_t *s, int n)
{
    uint8_t b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) b[j] = j < n ? __ldg(s + j) : (uint8_t)0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (j < n) ring[(o + j) & kMask1] = b[j];
}

// Output byte x, x < the window's start: from the ring when it is still
// held there (x >= lo), else from global memory.
__device__ __forceinline__ uint8_t out_byte(const uint8_t *ring, const uint8_t *src, const uint8_t *dst,
                                            const LzHole &h, int x, int lo)
{
    return x >= lo ? ring[x & kMask1] : old_byte(src, dst, h, x);
}

// ml <= 8 bytes of a match at ms whose sources lie before the window and
// in the ring; r runs through the source positions modulo off.
__device__ __forceinline__ void copy_match(uint8_t *ring, int ms, int off, int ml)
{
    uint8_t b[8];
    int r = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        b[j] = j < ml ? ring[(ms - off + r) & kMask1] : (uint8_t)0;
        r = r + 1 == off ? 0 : r + 1;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (j < ml) ring[(ms + j) & kMask1] = b[j];
}

// ml <= 8 bytes of a match at ms whose sources all lie before lo (in global
// memory, or in the input where the hole is); r as in copy_match.
__device__ __forceinline__ void copy_match_old(uint8_t *ring, int ms, int off, int ml, const uint8_t *src,
                                               const uint8_t *dst, const LzHole &h)
{
    uint8_t b[8];
    int r = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        b[j] = j < ml ? old_byte(src, dst, h, ms - off + r) : (uint8_t)0;
        r = r + 1 == off ? 0 : r + 1;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (j < ml) ring[(ms + j) & kMask1] = b[j];
}

__global__ void __launch_bounds__(128)
lz4_decode_kernel(const uint8_t *__restrict__ in, const long long *in_off, const int *in_len, int nchunks,
                  uint8_t *__restrict__ out, const long long *out_off, const int *out_cap, int *out_len,
                  int4 *hole, long long cap)
{
    __shared__ int4 cand_all[4][kWin];           // (literal start, literal length, match length, flags)
    __shared__ int next_all[4][kWin];            // input position after the candidate's sequence
    __shared__ __align__(16) uint8_t jump_all[4][5][kWin + 4];  // T_b; kExit: leaves the window
    __shared__ __align__(16) uint8_t ring_all[4][kRing1 + 16];  // recent output (16 bytes of slack)
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int4 *cand = cand_all[wib];
    int *nextp = next_all[wib];
    uint8_t(*T)[kWin + 4] = jump_all[wib];
    uint8_t *ring = ring_all[wib];
    if (lane < 4) {
#pragma unroll
        for (int b = 0; b < 5; ++b) T[b][kWin + lane] = (uint8_t)kExit;
    }
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int c = gw; c < nchunks; c += nw) {
        const uint8_t *src = in + in_off[c];
        const int iend = chunk_len(in_off, in_len, c);
        uint8_t *dst = out + (out_off ? out_off[c] : c * cap);
        const int oend = out_off ? out_cap[c] : (int)cap;
        int s0 = 0, op = 0, err = 0, ring_lo = 0;  // output before ring_lo is not in the ring
        bool done = false;
        LzHole hl;
        if (hole && lane == 0) hole[c] = make_int4(0, 0, 0, 0);  // written for every chunk
        // a literal run of n bytes from input i to output o, except the
        // record's byte planes 1 and 2 when it covers them whole (hole
        // given, record chunks: the record's byte count is output bytes 0-3)
        auto lit_run = [&](int o, int i, int n) {
            int a = 0, b = 0;
            if (hole && hl.len == 0 && o >= 4) {
                const int nb = (int)__ldcg(dst) | (int)__ldcg(dst + 1) << 8 | (int)__ldcg(dst + 2) << 16 |
                               (int)__ldcg(dst + 3) << 24;
                if (nb >= 4096 && nb <= 4096 + 4 * 32768 && ((nb - 4096) & 3) == 0) {
                    const int S = (nb - 4096) >> 2;
                    a = 4 + 4096 + S;
                    b = a + 2 * S;
                    if (!(o <= a && o + n >= b && b - a >= kMinHole)) a = b = 0;
                }
            }
            if (b > a) {
                warp_copy(dst + o, src + i, a - o, lane);
                warp_copy(dst + b, src + i + (b - o), o + n - b, lane);
                hl.out = a;
                hl.len = b - a;
                hl.in = i + (a - o);
                if (lane == 0) hole[c] = make_int4(hl.out, hl.in, hl.len, 0);
            } else {
                warp_copy(dst + o, src + i, n, lane);
            }
        };
        if (iend <= 0) {
            if (lane == 0) out_len[c] = 0;  // lz4.c:836: error exit at position 0
            continue;
        }
        while (!done && !err) {
            // ---- candidates s0 + 4*lane + j; the next window's input into L1
            if (lane < 2 && s0 + kWin + 128 * lane < iend)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(src + s0 + kWin + 128 * lane));
            {  // phase-major over the 4 candidates, so that their loads overlap
                int tok[4], ip[4], lit[4], ml[4], nx[4];
                bool more[4], stat[4];  // stat: a plain sequence so far
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int p = s0 + 4 * lane + j;
                    tok[j] = p < iend ? (int)__ldg(src + p) : -1;
                    ip[j] = p + 1;
                    lit[j] = (tok[j] >> 4) & 15;
                    ml[j] = tok[j] & 15;
                    nx[j] = 0;
                }
                // literal length continuation (lz4.c:846-850): the first byte
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    more[j] = false;
                    if (tok[j] >= 0 && lit[j] == 15 && ip[j] < iend) {
                        const int e = __ldg(src + ip[j]);
                        ++ip[j];
                        lit[j] += e;
                        more[j] = e == 255;
                    }
                }
                // ... and the rare longer ones
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    stat[j] = tok[j] >= 0;
                    if (more[j]) stat[j] = get_len_fast(src, ip[j], iend, lit[j]);
                }
                int flags[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    flags[j] = 0;
                    if (tok[j] >= 0) {
                        if (!stat[j]) flags[j] = kSlow;
                        else if (lit[j] > iend - ip[j] - (2 + 1 + kLastLiterals)) flags[j] = kTermIn;  // lz4.c:851
                    }
                    stat[j] = tok[j] >= 0 && flags[j] == 0;
                    if (stat[j]) nx[j] = ip[j] + lit[j] + 2;  // the offset is read for real sequences only
                }
                // match length continuation (lz4.c:873-882)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    more[j] = false;
                    if (stat[j] && ml[j] == 15 && nx[j] < iend - (kLastLiterals + 1)) {
                        const int e = __ldg(src + nx[j]);
                        ++nx[j];
                        ml[j] += e;
                        more[j] = e == 255;
                    }
                }
                uint32_t tword = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (more[j] && !get_len_fast(src, nx[j], iend - (kLastLiterals + 1), ml[j])) flags[j] = kSlow;
                    ml[j] += kMinMatch;
                    int t = kExit;
                    if (stat[j] && flags[j] == 0 && nx[j] - s0 < kWin) t = nx[j] - s0;
                    if (flags[j]) nx[j] = 0;
                    cand[4 * lane + j] = make_int4(ip[j], lit[j], ml[j], flags[j]);
                    nextp[4 * lane + j] = nx[j];
                    tword |= (uint32_t)t << (8 * j);
                }
                reinterpret_cast<uint32_t *>(T[0])[lane] = tword;
            }
            __syncwarp();
#pragma unroll
            for (int b = 1; b < 5; ++b) {
                const uint32_t w = reinterpret_cast<const uint32_t *>(T[b - 1])[lane];
                uint32_t v = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) v |= (uint32_t)T[b - 1][(w >> (8 * j)) & 0xff] << (8 * j);
                __syncwarp();
                reinterpret_cast<uint32_t *>(T[b])[lane] = v;
                __syncwarp();
            }
            // ---- lane k takes the k-th sequence of the chain
            int pos = 0;
#pragma unroll
            for (int b = 0; b < 5; ++b)
                if ((lane >> b) & 1) pos = T[b][pos];
            const bool member = pos < kWin;
            const int nm = __popc(__ballot_sync(0xffffffffu, member));
            int4 q = make_int4(0, 0, 0, 0);
            int nx = 0;
            if (member) {
                q = cand[pos];
                nx = nextp[pos];
            }
            const int flags = q.w & ~0xffff;
            const bool term_in = flags & kTermIn, slow = flags & kSlow;
            const int off = member && !term_in && !slow
                                ? (int)__ldg(src + q.x + q.y) | ((int)__ldg(src + q.x + q.y + 1) << 8)
                                : 0;
            int len = member && !slow ? q.y + (term_in ? 0 : q.z) : 0;
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int opl = op + incl - len, ms = opl + q.y;
            // ---- acceptance tests in sequence order (lz4.c:851-858, :868, :888-890)
            int stop = 0, epos = 0;  // 1: end of input, 2: malformed, 3: decode serially
            if (member) {
                if (slow) {
                    stop = 3;
                } else if (term_in || q.y > oend - opl - kMfLimit) {
                    if (q.y > oend - opl || q.y != iend - q.x) {
                        stop = 2;
                        epos = q.x;
                    } else {
                        stop = 1;
                    }
                } else if (off == 0 || off > ms) {
                    stop = 2;
                    epos = q.x + q.y + 2;
                } else if (q.z > oend - ms - kLastLiterals) {
                    stop = 2;
                    epos = nx;
                }
            }
            const unsigned sb = __ballot_sync(0xffffffffu, stop != 0);
            int ks = sb ? __ffs(sb) - 1 : nm;  // first sequence not taken as a plain one
            int kstop = __shfl_sync(0xffffffffu, stop, ks & 31);
            const int kepos = __shfl_sync(0xffffffffu, epos, ks & 31);
            // the window's output is staged in shared memory: sequences that
            // do not fit go to the serial path
            const unsigned fb = __ballot_sync(0xffffffffu, member && incl > kStage1);
            if (fb && __ffs(fb) - 1 <= ks) {
                ks = __ffs(fb) - 1;
                kstop = 3;
            }
            // sequences [0, ks) are complete; sequence ks contributes its
            // literals when it ends the input
            const bool lits = lane < ks || (lane == ks && kstop == 1);
            const bool mat = lane < ks;
            if (lits && q.y <= 8) copy_lit(ring, opl, src + q.x, q.y);
            unsigned pend = __ballot_sync(0xffffffffu, lits && q.y > 8);
            while (pend) {
                const int who = __ffs(pend) - 1;
                pend &= pend - 1;
                const int o0 = __shfl_sync(0xffffffffu, opl, who);
                const int x0 = __shfl_sync(0xffffffffu, q.x, who);
                const int n0 = __shfl_sync(0xffffffffu, q.y, who);
                for (int k = lane; k < n0; k += 32) ring[(o0 + k) & kMask1] = __ldg(src + x0 + k);
            }
            // matches whose sources lie before the window and are still in
            // the ring are copied by their lane; then, in rounds, every
            // short match whose source ends before the output of the first
            // match still to do (so that all of it is written) is copied by
            // its lane, and when there is none, that first match replays
            // with the whole warp (long matches, sources in global memory)
            const int lo = max(ring_lo, op + kStage1 - kRing1);  // not overwritten by this window
            const bool fast_ring = mat && q.z <= 8 && ms - off + min(q.z, off) <= op && ms - off >= lo;
            const bool fast_old = mat && q.z <= 8 && ms - off + min(q.z, off) <= lo;
            const bool fast = fast_ring || fast_old;
            if (fast_ring) copy_match(ring, ms, off, q.z);
            else if (fast_old) copy_match_old(ring, ms, off, q.z, src, dst, hl);
            __syncwarp();
            bool todo = mat && !fast;
            pend = __ballot_sync(0xffffffffu, todo);
            while (pend) {
                const int who = __ffs(pend) - 1;
                const int m0 = __shfl_sync(0xffffffffu, ms, who);
                const bool ready = todo && q.z <= 8 && ms - off + min(q.z, off) <= m0 && ms - off >= lo;
                const unsigned rb = __ballot_sync(0xffffffffu, ready);
                if (rb) {  // includes `who` when it is short with its source in the ring
                    if (ready) {
                        copy_match(ring, ms, off, q.z);
                        todo = false;
                    }
                    pend &= ~rb;
                } else {
                    pend &= pend - 1;
                    if (lane == who) todo = false;
                    const int o0 = __shfl_sync(0xffffffffu, off, who);
                    const int l0 = __shfl_sync(0xffffffffu, q.z, who);
                    for (int k = lane; k < l0; k += 32) {
                        const int x = m0 - o0 + msrc(k, o0, l0);
                        ring[(m0 + k) & kMask1] = out_byte(ring, src, dst, hl, x, lo);
                    }
                }
                __syncwarp();
            }
            const int nout = kstop == 1 ? __shfl_sync(0xffffffffu, opl + q.y, ks & 31) - op
                                        : (ks > 0 ? __shfl_sync(0xffffffffu, incl, ks - 1) : 0);
            {
                const int r = op & kMask1, n1 = min(nout, kRing1 - r);
                flush(dst + op, ring, r, n1, lane, 32);
                if (nout > n1) flush(dst + op + n1, ring, 0, nout - n1, lane, 32);
            }
            __syncwarp();
            // ---- advance
            op += nout;
            if (kstop == 1) {
                done = true;
            } else if (kstop == 2) {
                err = kepos;
            } else if (kstop == 3) {
                // a sequence with long length fields, decoded serially
                int ip = __shfl_sync(0xffffffffu, s0 + pos, ks & 31);
                const int token = src[ip++];
                long long ll = token >> 4;
                if (ll == 15) ll += get_len(src, ip, iend, lane);
                if (ll > (long long)(oend - op - kMfLimit) || ll > (long long)(iend - ip - (2 + 1 + kLastLiterals))) {
                    if (ll > (long long)(oend - op) || ll != (long long)(iend - ip)) {
                        err = ip;
                    } else {
                        lit_run(op, ip, (int)ll);
                        op += (int)ll;
                        done = true;
                    }
                } else {
                    lit_run(op, ip, (int)ll);
                    op += (int)ll;
                    ip += (int)ll;
                    const int o = (int)src[ip] | ((int)src[ip + 1] << 8);
                    ip += 2;
                    if (o == 0 || o > op) {
                        err = ip;
                    } else {
                        long long m = token & 15;
                        if (m == 15) m += get_len(src, ip, iend - (kLastLiterals + 1), lane);
                        m += kMinMatch;
                        if (m > (long long)(oend - op - kLastLiterals)) {
                            err = ip;
                        } else {
                            __syncwarp();
                            for (int k = lane; k < (int)m; k += 32)
                                dst[op + k] = old_byte(src, dst, hl, op - o + msrc(k, o, (int)m));
                            __syncwarp();
                            op += (int)m;
                            s0 = ip;
                            ring_lo = op;  // written around the ring
                        }
                    }
                }
            } else {
                s0 = __shfl_sync(0xffffffffu, nx, nm - 1);
            }
            __syncwarp();
        }
        if (lane == 0) out_len[c] = err ? -err : op;
        __syncwarp();
    }
}

// gridDim.y CTAs per chunk: the chunk's bytes to dst + dst_off[c]. With `hole`
// (LZ4 of block records), bytes [hole.x, hole.x + hole.z) of the chunk's
// output are the input bytes at hsrc + hsrc_off[c] + hole.y, which the
// encoder left unwritten. SCAN: the chunk sums the lengths before its own and
// writes its offset (for chunk counts where that is cheaper than a launch).
template <bool SCAN>
__global__ void __launch_bounds__(256)
gather_kernel(const uint8_t *__restrict__ src, const long long *src_off, const int *len, int nchunks,
              uint8_t *__restrict__ dst, long long *dst_off, int *flag, long long *total, const int4 *hole,
              const uint8_t *__restrict__ hsrc, const long long *hsrc_off)
{
    const int c = blockIdx.x;
    const int n = len[c];
    long long at;
    if (SCAN) {
        __shared__ long long part[8];
        long long sum = 0;
        for (int i = threadIdx.x; i < c; i += 256) sum += len[i];
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
        __syncthreads();
        at = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) at += part[w];
        if (threadIdx.x == 0 && blockIdx.y == 0) dst_off[c] = at;
    } else {
        at = dst_off[c];
    }
    if (threadIdx.x == 0 && blockIdx.y == 0) {
        if (n < 0 && flag) atomicMin(flag, -1);
        if (c == nchunks - 1) {
            if (SCAN) dst_off[nchunks] = at + n;
            if (total) *total = at + n;
        }
    }
    if (n <= 0) return;
    // this CTA's part of the chunk
    const int share = gridDim.y == 1 ? n : ((n + (int)gridDim.y - 1) / (int)gridDim.y + 15) & ~15;
    const int lo = min(share * (int)blockIdx.y, n), hi = min(lo + share, n);
    const uint8_t *s = src + src_off[c];
    uint8_t *d = dst + at;
    const int4 hl = hole ? hole[c] : make_int4(0, 0, 0, 0);
    auto copy = [&](const uint8_t *from, int a, int b) {  // output bytes [a, b) from `from` + a
        a = max(a, lo);
        b = min(b, hi);
        if (b > a) cta_copy(d + a, from + a, b - a);
    };
    if (hl.z > 0) {
        copy(s, 0, hl.x);
        copy(hsrc + hsrc_off[c] + hl.y - hl.x, hl.x, hl.x + hl.z);
        copy(s, hl.x + hl.z, n);
    } else {
        copy(s, 0, n);
    }
}

}  // namespace cz

using namespace cz;

static int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) !=
                                                   cudaSuccess)
        sms = 1;
    return sms;
}


// kLzWarps chunks per CTA; 16 (512 threads, ~123 KB of shared memory)
// takes an SM, so that CTAs of this kernel and the wavelet kernel, which
// also takes a whole SM, share the machine SM by SM.
// Up to 9 chunks per SM: two warps per chunk. One-record chunks, ms with two
// warps / with one: 64 chunks 0.17 / 0.29, 512 0.23 / 0.33, 1 024 0.22 / 0.30,
// 2 048 0.30 / 0.27, 4 096 0.90 / 0.67 (there the warps fill the SMs either way
// and two need more registers); 128 chunks of 4 records 1.03 / 1.56, 69 of 15
// 2.99 / 4.30. The CTA width asked for only shapes the other kernel; 16, whole-SM
// CTAs that leave the other SMs free, is never taken over.

template <int W, bool SEQ, int E, int SW>
static cudaError_t launch_enc_t(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks,
                                uint8_t *out, const long long *out_off, int *out_len, int records, int grid,
                                cudaStream_t st, int4 *hole)
{
    if (W < 16 && nchunks <= kLzPairChunksPerSm * sm_count()) {
        lz4_encode_pair_kernel<SEQ, E, SW>
            <<<nchunks, 64, 0, st>>>(in, in_off, in_len, nchunks, out, out_off, out_len, records, hole);
        return cudaGetLastError();
    }
    const int sm = W <= 8 ? 0 : (int)sizeof(LzEncWarp<SW, (E >= 2)>) * W;
    auto k = lz4_encode_kernel<W, SEQ, E, SW>;
    if (sm > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (e != cudaSuccess) return e;
    }
    k<<<grid, W * 32, sm, st>>>(in, in_off, in_len, nchunks, out, out_off, out_len, records, hole);
    return cudaGetLastError();
}

// one kernel per effort level, so that a level pays only for its own work
template <int W, bool SEQ, int SW>
static cudaError_t launch_enc_e(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks,
                                uint8_t *out, const long long *out_off, int *out_len, int records, int grid,
                                cudaStream_t st, int4 *hole, int effort)
{
    switch (effort) {
    case 0:
        return launch_enc_t<W, SEQ, 0, SW>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st,
                                           hole);
    case 2:
        return launch_enc_t<W, SEQ, 2, SW>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st,
                                           hole);
    default:
        return launch_enc_t<W, SEQ, 1, SW>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st,
                                           hole);
    }
}

// The super-window size depends only on the chunk count and the GPU, so
// that every CTA width writes the same bytes: 768 positions when all chunks
// fit on the SMs at once with 4 chunks per CTA (7 CTAs of 4 warps per SM),
// else 512.
static int window_for(int nchunks) { return (long long)nchunks <= 28LL * sm_count() ? kWinLarge : kWinSmall; }

template <int W, bool SEQ>
static cudaError_t launch_enc(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks,
                              uint8_t *out, const long long *out_off, int *out_len, int records, int grid,
                              cudaStream_t st, int4 *hole, int effort)
{
    if (window_for(nchunks) == kWinLarge)
        return launch_enc_e<W, SEQ, kWinLarge>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st,
                                               hole, effort);
    return launch_enc_e<W, SEQ, kWinSmall>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st,
                                           hole, effort);
}

cudaError_t cz_launch_lz4_encode(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks,
                                 uint8_t *out, const long long *out_off, int *out_len, int records, int warps,
                                 int grid, cudaStream_t st, int4 *hole, int effort)
{
    if (nchunks <= 0) return cudaSuccess;
    switch (warps) {
    case 2:
        return launch_enc<2, false>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st, hole, effort);
    case 8:
        return launch_enc<8, false>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st, hole, effort);
    case 16:
        return launch_enc<16, false>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st, hole, effort);
    default:
        return launch_enc<4, false>(in, in_off, in_len, nchunks, out, out_off, out_len, records, grid, st, hole, effort);
    }
}

cudaError_t cz_launch_lz77_parse(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks,
                                 uint8_t *seq, const long long *seq_off, int *seq_bytes, int records, int grid,
                                 cudaStream_t st, int effort)
{
    if (nchunks <= 0) return cudaSuccess;
    return launch_enc<4, true>(in, in_off, in_len, nchunks, seq, seq_off, seq_bytes, records, grid, st, nullptr, effort);
}

// A CTA per chunk finishes a chunk 3 to 4 times sooner than a warp, but
// executes about 1.5 times the instructions: it is the faster one until the
// warps of one-warp chunks fill the SMs. Measured (ms, CTA / warp per chunk):
// 512 chunks of a 256^3 field 0.36 / 0.59, 1 024 of 256x256x512 0.38 / 0.46,
// 1 728 of 384^3 0.71 / 0.56, 2 048 of 256x512x512 0.51 / 0.39; 274 chunks
// of 15 records 2.03 / 7.24, 1 024 of 4 records 1.58 / 2.13.
constexpr int kWideChunksPerSm = 8;

cudaError_t cz_launch_lz4_decode(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks,
                                 uint8_t *out, const long long *out_off, const int *out_cap, int *out_len,
                                 cudaStream_t st, int4 *hole, long long cap)
{
    if (nchunks <= 0) return cudaSuccess;
    const int sms = sm_count();
    if (nchunks <= kWideChunksPerSm * sms) {
        const int sm = (int)sizeof(LzDecShared);
        const cudaError_t e =
            cudaFuncSetAttribute(lz4_decode_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (e != cudaSuccess) return e;
        lz4_decode_wide_kernel<<<std::min(nchunks, 3 * sms), kDecThreads, sm, st>>>(in, in_off, in_len, nchunks, out,
                                                                                   out_off, out_cap, out_len, hole, cap);
    } else {
        lz4_decode_kernel<<<std::min((nchunks + 3) / 4, 8 * sms), 128, 0, st>>>(in, in_off, in_len, nchunks, out, out_off,
                                                                               out_cap, out_len, hole, cap);
    }
    return cudaGetLastError();
}

cudaError_t cz_launch_gather(const uint8_t *src, const long long *src_off, const int *len, int nchunks,
                             uint8_t *dst, long long *dst_off, bool scan, int *flag, long long *total,
                             cudaStream_t st, const int4 *hole, const uint8_t *hsrc, const long long *hsrc_off)
{
    if (nchunks <= 0) return cudaSuccess;
    // summed per chunk up to 1024 chunks: at most 4 KB of lengths per CTA
    // (a scan launch of its own costs 4 us)
    const bool own = scan && nchunks <= 1024;
    if (scan && !own) {
        cudaError_t e = cudaMemsetAsync(dst_off, 0, sizeof(long long), st);
        if (e == cudaSuccess) e = cz_launch_scan_from(len, nchunks, dst_off, st);
        if (e != cudaSuccess) return e;
    }
    // a CTA moves 4 KB per round trip to memory: few chunks go to several CTAs
    // (64 raw records 12 -> 6 us), unless the other streams' kernels share the GPU
    const int parts = scan ? std::max(1, std::min(8, 8 * sm_count() / nchunks)) : 1;
    auto k = own ? gather_kernel<true> : gather_kernel<false>;
    k<<<dim3(nchunks, parts), 256, 0, st>>>(src, src_off, len, nchunks, dst, dst_off, flag, total, hole, hsrc, hsrc_off);
    return cudaGetLastError();
}
