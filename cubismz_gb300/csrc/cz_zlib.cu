// cz_zlib.cu -- zlib streams (RFC 1950 wrapper, RFC 1951 DEFLATE), the
// format of the reference's zlib encoder (deflateInit/deflate with Z_FINISH,
// CompressionEncoders.h:116-190) and decoder (inflateInit/inflate,
// CompressionEncoders.h:48-88).
//
// Encoder (deflate_kernel): one CTA per chunk, a warp per DEFLATE block, fed by
// the LZ77 parse of the LZ4 encoder run with a 32 KiB window (cz_lz4.cu, SEQ
// mode). A chunk of shuffled block records gets a DEFLATE block per record mask
// and byte plane (other chunks one per 64 KiB): per block, the warp counts the
// symbols of the items that start in it (literal bytes; matches of more than
// 258 bytes in pieces), sorts the used symbols (bitonic, by frequency), builds
// the length-limited codes (cz_deflate.cuh), and the exact sizes of the
// stored, fixed and dynamic codings pick the smallest; then 32 sequences per
// step, a warp scan of their bit counts, and OR-writes into a per-warp ring of
// words that is flushed to the output with word stores. zlib header 78 9C,
// Adler-32 by a reduction.
//
// Decoder (inflate_kernel): two warps per chunk, because a DEFLATE stream is
// one serial chain of bits and that chain is what bounds it. Lane 0 of the
// first warp does nothing but decode: headers, and symbols from lookup tables
// (which the whole warp builds) into records of up to six literals and a
// match, without a look at positions, limits or bytes. The second warp takes
// 32 records at a time: a scan gives their output positions, every test is
// made there, literals and matches go to a ring in shared memory (a match per
// lane as soon as its source is written) that is flushed with word stores.
// Stored blocks are copied by the warp. The Adler-32 of the output is a sum
// over both warps, checked against the trailer. Malformed input (bad header,
// code lengths, symbols, distances past the start, output past the capacity,
// truncated input or a wrong checksum) gives a negative length; every read and
// write is bounds checked. Zlib stage of
// 512 one-record chunks (256^3): 10.2 -> 3.6 ms; a record of the queue takes
// about 360 cycles, 70 dependent instructions of one lane.
#include "cz_bytes.cuh"
#include "cz_codec.h"
#include "cz_deflate.cuh"

namespace cz {

using namespace zl;

constexpr int kZBatch = 128;  // records per batch
// The ring holds what 32 records can add (six literals and a match of 258
// bytes each) and at least 7 KB of history; older sources come from the output.
constexpr int kZRing = 16384, kZRingM = kZRing - 1, kZGroup = 32 * (6 + 258);

// n bytes from s to d by the warp (4-byte stores once d is aligned); every
// load is of an aligned word holding at least one byte of the run.
__device__ __forceinline__ void run_copy(uint8_t *d, const uint8_t *s, int n, int lane)
{
    int h = (int)((4 - (reinterpret_cast<uintptr_t>(d) & 3)) & 3);
    if (h > n) h = n;
    if (lane < h) d[lane] = s[lane];
    d += h;
    s += h;
    n -= h;
    const int nw = n >> 2;
    const uint32_t sa = (uint32_t)(reinterpret_cast<uintptr_t>(s) & 3);
    const uint32_t *sw = reinterpret_cast<const uint32_t *>(s - sa);
    uint32_t *dw = reinterpret_cast<uint32_t *>(d);
    for (int i = lane; i < nw; i += 32) dw[i] = sa ? __funnelshift_r(sw[i], sw[i + 1], 8 * sa) : sw[i];
    const int t = n & 3;
    if (lane < t) d[4 * nw + lane] = s[4 * nw + lane];
}

// Adler-32 sums of n bytes at d (4-byte aligned) by threads t of nt: the sum
// of the bytes and of (n - i) times byte i. CG: read past L1 (bytes the
// kernel wrote).
template <bool CG>
__device__ __forceinline__ void adler_sums(const uint8_t *d, int n, int t, int nt, unsigned long long &sa,
                                           unsigned long long &sb)
{
    const uint32_t *w = reinterpret_cast<const uint32_t *>(d);
    sa = sb = 0;
    const int nw = n >> 2;
#pragma unroll 8
    for (int i = t; i < nw; i += nt) {
        const uint32_t v = CG ? __ldcg(w + i) : w[i];
        const unsigned s = __dp4a(v, 0x01010101u, 0u);
        sa += s;
        sb += (unsigned long long)(unsigned)(n - 4 * i) * s - __dp4a(v, 0x03020100u, 0u);
    }
    const int i = 4 * nw + t;
    if (i < n) {
        const unsigned v = CG ? __ldcg(d + i) : d[i];
        sa += v;
        sb += (unsigned long long)(n - i) * v;
    }
}
__device__ __forceinline__ unsigned adler_of(unsigned long long sa, unsigned long long sb, int n)
{
    return ((unsigned)(((unsigned long long)n + sb) % 65521ull) << 16) | (unsigned)((1 + sa) % 65521ull);
}

// zl::build by the warp. cnt: 2 x 16 words of scratch.
__device__ bool warp_build(Huff &h, const unsigned char *len, int n, bool lit, unsigned *cnt, int lane)
{
    if (lane < 16) cnt[lane] = 0;
    __syncwarp();
    for (int s = lane; s < n; s += 32)
        if (len[s]) atomicAdd(&cnt[len[s]], 1u);
    __syncwarp();
    if (lane < 16) h.count[lane] = (unsigned short)cnt[lane];
    __syncwarp();
    if (!lengths_ok(h.count, false)) return false;
    // first code and symbol offset of every length (lane l: length l)
    unsigned first = 0, offs = 0, code = 0, sum = 0;
    for (int l = 1; l <= kMaxBits; ++l) {
        code = (code + (l > 1 ? cnt[l - 1] : 0u)) << 1;
        if (lane == l) {
            first = code;
            offs = sum;
        }
        sum += cnt[l];
    }
    __syncwarp();
    if (lane < 16) cnt[16 + lane] = offs;  // next place per length
    if (lane >= 1 && lane <= kMaxBits) {
        h.lim[lane] = (unsigned short)((first + cnt[lane]) << (kMaxBits - lane));
        h.shift[lane] = (short)((int)offs - (int)first);
    }
    __syncwarp();
    for (int s0 = 0; s0 < n; s0 += 32) {  // symbols in order
        const int s = s0 + lane, l = s < n ? len[s] : 0;
        const unsigned same = __match_any_sync(0xffffffffu, l);
        const int rank = __popc(same & ((1u << lane) - 1u));
        const unsigned at = cnt[16 + l];
        if (l) h.sym[at + rank] = (unsigned short)s;
        __syncwarp();
        if (l && rank == 0) cnt[16 + l] = at + __popc(same);
        __syncwarp();
    }
    // the table by index: a code of length l is the smallest l whose codes
    // end above the index's first l bits (canonical codes grow with length)
    unsigned lim[kFastBits + 1], shift[kFastBits + 1];  // per length: end of its codes on kFastBits bits; symbol - code
#pragma unroll
    for (int l = 1; l <= kFastBits; ++l) {
        const unsigned f = __shfl_sync(0xffffffffu, first, l);
        lim[l] = (f + cnt[l]) << (kFastBits - l);
        shift[l] = __shfl_sync(0xffffffffu, offs, l) - f;
    }
#pragma unroll 1
    for (int i = lane; i < 1 << kFastBits; i += 32) {
        const unsigned v = __brev((unsigned)i) >> (32 - kFastBits);
        int l = 0;
        unsigned at = 0;
#pragma unroll
        for (int k = kFastBits; k >= 1; --k)
            if (v < lim[k]) {
                l = k;
                at = (v >> (kFastBits - k)) + shift[k];
            }
        unsigned e = 0;
        if (l) {
            const int s = h.sym[at];
            e = lit ? lit_entry(s, l) : dist_entry(s, l);
        }
        h.fast[i] = e;
    }
    __syncwarp();
    if (lit) {
        // a combined entry keeps its first literal, so any order will do
        for (int i = lane; i < 1 << kFastBits; i += 32) h.fast[i] = pair_entry(h.fast, i);
        __syncwarp();
    }
    return true;
}

template <int ID>
__device__ __forceinline__ void bar_arrive64()
{
    asm volatile("bar.arrive %0, 64;" ::"n"(ID) : "memory");
}
template <int ID>
__device__ __forceinline__ void bar_sync64()
{
    asm volatile("bar.sync %0, 64;" ::"n"(ID) : "memory");
}

__global__ void __launch_bounds__(64, 7)
inflate_kernel(const uint8_t *__restrict__ in, const long long *in_off, const int *in_len, int nchunks,
               uint8_t *__restrict__ out, const long long *out_off, const int *out_cap, int *out_len, long long cap)
{
    __shared__ Huff lit, dist;
    __shared__ unsigned char lens[320];
    __shared__ unsigned scratch[32];
    __shared__ uint4 queue[2][kZBatch];  // records
    __shared__ int s_state[2][4];        // per batch: records, last one of the chunk, a stored block's input position and bytes
    __shared__ int s_end[4];             // error of the decoder and of the writer, Adler-32 of the trailer, output size
    __shared__ unsigned long long s_sum[2];
    __shared__ __align__(16) uint8_t ring[kZRing + 16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint8_t *src = in + in_off[c];
        const long long span = in_len ? in_len[c] : in_off[c + 1] - in_off[c];
        const int nin = span < 0 || span > 0x7fffffffLL ? -1 : (int)span;
        uint8_t *dst = out + (out_off ? out_off[c] : c * cap);
        const int oend = out_off ? out_cap[c] : (int)cap;
        // barriers 1, 2: batch k is full; 3, 4: batch k is free again
        if (warp == 0) {
            Inflater z;  // lane 0's decoder state, kept in registers
            if (lane == 0) z.start(src, nin);
            uint32_t it = 0;
            for (int last = 0; !last; ++it) {
                const int k = it & 1;
                if (it >= 2) {
                    if (k) bar_sync64<4>();
                    else bar_sync64<3>();
                }
                int n = 0, want = 0;
                if (lane == 0) z.run_n = 0;
                do {
                    want = 0;
                    if (lane == 0) {
                        while (!z.err && n < kZBatch) {
                            if (!z.in_block) {
                                if (z.final_block || z.block_header(lit.fast, lens)) break;
                                if (z.btype != 0) {
                                    want = z.nlen | z.ndist << 16;
                                    break;
                                }
                                (void)z.stored_run();
                                break;
                            }
                            while (n < kZBatch && z.in_block && !z.err) {
                                const Record r = z.record(lit, dist);
                                queue[k][n++] = make_uint4(r.e[0], r.e[1], r.e[2], r.m);
                            }
                            if (!z.err && z.b.over()) z.err = 14;
                        }
                    }
                    __syncwarp();
                    want = __shfl_sync(0xffffffffu, want, 0);
                    if (want) {
                        const int nlen = want & 0xffff, ndist = want >> 16;
                        const bool ok = warp_build(lit, lens, nlen, true, scratch, lane);
                        const bool ok2 = ok && warp_build(dist, lens + nlen, ndist, false, scratch, lane);
                        if (lane == 0 && !ok2) z.err = ok ? 10 : 9;
                        __syncwarp();
                    }
                } while (want);
                if (lane == 0) {
                    last = z.err || z.done();
                    if (last) {
                        if (!z.err) s_end[2] = (int)z.trailer();
                        s_end[0] = z.err;
                    }
                    s_state[k][0] = n;
                    s_state[k][1] = last;
                    s_state[k][2] = (int)z.run_src;
                    s_state[k][3] = (int)z.run_n;
                }
                last = __shfl_sync(0xffffffffu, last, 0);
                if (k) bar_arrive64<2>();
                else bar_arrive64<1>();
            }
            // every batch is written before the chunk ends
            for (uint32_t j = it < 2 ? 0 : it - 2; j < it; ++j) {
                if (j & 1) bar_sync64<4>();
                else bar_sync64<3>();
            }
        } else {
            int op = 0, ring_lo = 0, err = 0;  // output before ring_lo is not in the ring
            for (uint32_t it = 0, last = 0; !last; ++it) {
                const int kb = it & 1;
                if (kb) bar_sync64<2>();
                else bar_sync64<1>();
                const int n = s_state[kb][0];
                last = (uint32_t)s_state[kb][1];
                for (int i0 = 0; i0 < n && !err; i0 += 32) {
                    const uint4 r = i0 + lane < n ? queue[kb][i0 + lane] : make_uint4(0, 0, 0, 0);
                    const int c0 = literals(r.x), c1 = literals(r.y), c2 = literals(r.z);
                    const int nl = c0 + c1 + c2 + (int)(r.w >> 31);
                    const int len = r.w >> 31 ? 0 : (int)(r.w & 511u), d = len ? (int)(r.w >> 9) : 1;
                    int incl = nl + len;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    const int total = __shfl_sync(0xffffffffu, incl, 31);
                    const int at = op + incl - nl - len, p = at + nl;  // the record's literals, its match
                    // against the room left: with a capacity near 2^31 the ends
                    // themselves may not be ints
                    const int room = oend - op;
                    const int bad = incl - len > room ? 15 : len && d > p ? 19 : incl > room ? 20 : 0;
                    const unsigned bb = __ballot_sync(0xffffffffu, bad != 0);
                    if (bb) {
                        err = __shfl_sync(0xffffffffu, bad, __ffs(bb) - 1);
                        break;
                    }
                    const int a1 = at + c0, a2 = a1 + c1;
                    if (c0 > 0) ring[at & kZRingM] = (uint8_t)(r.x >> 8);
                    if (c0 > 1) ring[(at + 1) & kZRingM] = (uint8_t)(r.x >> 16);
                    if (c1 > 0) ring[a1 & kZRingM] = (uint8_t)(r.y >> 8);
                    if (c1 > 1) ring[(a1 + 1) & kZRingM] = (uint8_t)(r.y >> 16);
                    if (c2 > 0) ring[a2 & kZRingM] = (uint8_t)(r.z >> 8);
                    if (c2 > 1) ring[(a2 + 1) & kZRingM] = (uint8_t)(r.z >> 16);
                    if (r.w >> 31) ring[(p - 1) & kZRingM] = (uint8_t)r.w;
                    __syncwarp();
                    // matches in rounds: every one whose source ends before the
                    // output of the first one still to do (so that all of it is
                    // written) is copied by its lane, long ones by the warp; the
                    // first one itself always is. Byte k is out[p - d + (k mod d)].
                    const int lo = max(ring_lo, op + kZGroup - kZRing);  // not overwritten by this group
                    auto from = [&](int x) -> uint8_t { return x >= lo ? ring[x & kZRingM] : __ldcg(dst + x); };
                    const int send = p - d + min(len, d);
                    unsigned todo = __ballot_sync(0xffffffffu, len > 0);
                    while (todo) {
                        const int m0 = __shfl_sync(0xffffffffu, p, __ffs(todo) - 1);
                        const bool go = (todo >> lane & 1u) && send <= m0;
                        if (go && len <= 32) {
                            int x = p - d;
                            for (int k = 0; k < len; k += 4) {
                                uint8_t v[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    v[j] = k + j < len ? from(x) : (uint8_t)0;
                                    if (++x == p) x = p - d;
                                }
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    if (k + j < len) ring[(p + k + j) & kZRingM] = v[j];
                            }
                        }
                        for (unsigned lng = __ballot_sync(0xffffffffu, go && len > 32); lng; lng &= lng - 1) {
                            const int who = __ffs(lng) - 1;
                            const int pp = __shfl_sync(0xffffffffu, p, who), ll = __shfl_sync(0xffffffffu, len, who);
                            const int dd = __shfl_sync(0xffffffffu, d, who);
                            for (int k = lane; k < ll; k += 32)
                                ring[(pp + k) & kZRingM] = from(pp - dd + (dd >= ll ? k : k % dd));
                        }
                        todo &= ~__ballot_sync(0xffffffffu, go);
                        __syncwarp();
                    }
                    const int r0 = op & kZRingM, n1 = min(total, kZRing - r0);
                    flush(dst + op, ring, r0, n1, lane, 32);
                    if (total > n1) flush(dst + op + n1, ring, 0, total - n1, lane, 32);
                    op += total;
                    __syncwarp();
                }
                const int rn = s_state[kb][3];
                if (rn > 0 && !err) {
                    if (rn > oend - op) {
                        err = 12;
                    } else {
                        run_copy(dst + op, src + s_state[kb][2], rn, lane);
                        op += rn;
                        ring_lo = op;  // written around the ring
                    }
                }
                if (last && lane == 0) {
                    s_end[1] = err;
                    s_end[3] = op;
                }
                if (kb) bar_arrive64<4>();
                else bar_arrive64<3>();
            }
        }
        __syncthreads();
        // Adler-32 of the output (A = 1 + sum d_i, B = n + sum (n - i) d_i,
        // mod 65521) against the trailer
        int e = s_end[0] ? s_end[0] : s_end[1];
        const int total = s_end[3];
        if (!e) {
            unsigned long long sa, sb;
            adler_sums<true>(dst, total, threadIdx.x, 64, sa, sb);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sa += __shfl_xor_sync(0xffffffffu, sa, o);
                sb += __shfl_xor_sync(0xffffffffu, sb, o);
            }
            if (threadIdx.x == 32) {
                s_sum[0] = sa;
                s_sum[1] = sb;
            }
            __syncthreads();
            if (threadIdx.x == 0 && adler_of(sa + s_sum[0], sb + s_sum[1], total) != (unsigned)s_end[2]) e = 22;
        }
        if (threadIdx.x == 0) out_len[c] = e ? -e : total;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- encoder
constexpr int kZWarps = 5;     // warps per chunk: a record's mask and byte planes are five blocks
constexpr int kRingW = 1024;   // bit-ring words per warp: 32 short sequences fit (see block_items)
constexpr int kRingM = kRingW - 1;

struct DeflateWarp {
    uint32_t lf[288], df[32];
    Codes codes;
    union {
        uint32_t ring[kRingW];
        struct {  // code construction
            uint32_t key[512];  // (weight << 9 | symbol), sorted; unused: ~0
            uint32_t w[288], iw[288];
            uint16_t sym[288], par[576], dep[576];
            uint8_t l[288];
        } b;
    } u;
    uint32_t cnt[32];  // scratch of the code construction
};

// zl::huff_lengths of the n sorted weights in s.u.b.w into s.u.b.l, by the
// warp: lane 0 only merges (both queues' heads in registers) and takes the
// depths of the internal nodes; leaves, counts and lengths are shared out.
__device__ bool warp_huff_lengths(DeflateWarp &s, int n, int maxbits, int lane)
{
    auto &b = s.u.b;
    if (lane < 16) s.cnt[lane] = 0;
    if (lane == 0) {
        constexpr uint32_t kNone = 0xffffffffu;
        int i = 0, j = 0;
        uint32_t wi = b.w[0], wj = kNone;  // next leaf, next internal node (block counts stay below 2^22)
        for (int k = 0; k < n - 1; ++k) {
            uint32_t sum = 0;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (wi <= wj) {  // a leaf goes first among equals, as there is one
                    b.par[i++] = (uint16_t)(n + k);
                    sum += wi;
                    wi = i < n ? b.w[i] : kNone;
                } else {
                    b.par[n + j++] = (uint16_t)(n + k);
                    sum += wj;
                    wj = j < k ? b.iw[j] : kNone;
                }
            }
            b.iw[k] = sum;
            if (j == k) wj = sum;
        }
        b.dep[2 * n - 2] = 0;
        for (int x = 2 * n - 3; x >= n; --x) b.dep[x] = (uint16_t)(b.dep[b.par[x]] + 1);  // parents come later
    }
    __syncwarp();
    for (int x = lane; x < n; x += 32) atomicAdd(&s.cnt[min((int)b.dep[b.par[x]] + 1, maxbits)], 1u);
    __syncwarp();
    int ok = 1;
    if (lane == 0) {
        uint32_t kraft = 0, total = 0;
        for (int l = 1; l <= maxbits; ++l) kraft += s.cnt[l] << (maxbits - l);
        while (kraft > (1u << maxbits)) {
            int l = maxbits - 1;
            while (l > 0 && s.cnt[l] == 0) --l;
            if (l == 0 || s.cnt[maxbits] == 0) {
                ok = 0;
                break;
            }
            s.cnt[maxbits]--;
            s.cnt[l]--;
            s.cnt[l + 1] += 2;
            --kraft;
        }
        for (int l = 1; l <= maxbits; ++l) total += s.cnt[l];
        ok = ok && kraft == (1u << maxbits) && (int)total == n;
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    if (!ok) return false;
    for (int x = lane; x < n; x += 32) {  // longest first
        int l = maxbits, end = (int)s.cnt[maxbits];
        while (x >= end) end += (int)s.cnt[--l];
        b.l[x] = (uint8_t)l;
    }
    __syncwarp();
    return true;
}

// Code lengths for freq[0..n) into len: the warp sorts the used symbols by
// (frequency, symbol) -- a bitonic sort of keys weight << 9 | symbol over 512
// slots, 32 for the distance code (block counts stay below 2^22). False if it
// fails.
__device__ bool warp_code(DeflateWarp &s, const uint32_t *freq, int n, uint8_t *len, int lane)
{
    auto &b = s.u.b;
    int used = 0;
    for (int x = lane; x < n; x += 32) used += freq[x] != 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) used += __shfl_xor_sync(0xffffffffu, used, o);
    // at least two codes: the lowest unused symbols get weight one (never sent)
    int need = used < 2 ? 2 - used : 0;
    const int slots = n <= 32 ? 32 : 512;
    for (int x0 = 0; x0 < slots; x0 += 32) {
        const int x = x0 + lane;
        uint32_t f = x < n ? freq[x] : 0u;
        const bool zero = x < n && f == 0u;
        const unsigned zb = __ballot_sync(0xffffffffu, zero);
        if (zero && need > 0 && __popc(zb & ((1u << lane) - 1u)) < need) f = 1u;
        need -= min(need, __popc(zb));
        b.key[x] = f ? (f << 9 | (uint32_t)x) : 0xffffffffu;
    }
    used = max(used, 2);
    __syncwarp();
    // bitonic sort, ascending, slots / 2 compare-exchanges per pass
    for (int k = 2; k <= slots; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll 4
            for (int i = lane; i < slots / 2; i += 32) {
                const int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1)), hi = lo + j;
                const uint32_t a = b.key[lo], c = b.key[hi];
                const bool up = (lo & k) == 0;
                if ((a > c) == up) {
                    b.key[lo] = c;
                    b.key[hi] = a;
                }
            }
            __syncwarp();
        }
    }
    for (int x = lane; x < n; x += 32) len[x] = 0;
    for (int r = lane; r < used; r += 32) {
        const uint32_t kk = b.key[r];
        b.sym[r] = (uint16_t)(kk & 511u);
        b.w[r] = kk >> 9;
    }
    __syncwarp();
    const bool ok = warp_huff_lengths(s, used, zl::kMaxLit, lane);
    if (ok)
        for (int i = lane; i < used; i += 32) len[b.sym[i]] = b.l[i];
    __syncwarp();
    return ok;
}

// zl::canon_codes by the warp: codes in symbol order per length.
__device__ void warp_canon_codes(DeflateWarp &s, const uint8_t *len, int n, uint16_t *code, int lane)
{
    if (lane < 16) s.cnt[lane] = 0;
    __syncwarp();
    for (int x = lane; x < n; x += 32)
        if (len[x]) atomicAdd(&s.cnt[len[x]], 1u);
    __syncwarp();
    uint32_t first = 0, c = 0;
    for (int l = 1; l < 16; ++l) {
        c = (c + (l > 1 ? s.cnt[l - 1] : 0u)) << 1;
        if (lane == l) first = c;
    }
    __syncwarp();
    if (lane < 16) s.cnt[lane] = first;  // next code per length
    __syncwarp();
    for (int x0 = 0; x0 < n; x0 += 32) {
        const int x = x0 + lane, l = x < n ? len[x] : 0;
        const unsigned same = __match_any_sync(0xffffffffu, l);
        const int rank = __popc(same & ((1u << lane) - 1u));
        const uint32_t at = s.cnt[l];
        if (x < n) code[x] = l ? (uint16_t)(__brev(at + rank) >> (32 - l)) : (uint16_t)0;
        __syncwarp();
        if (l && rank == 0) s.cnt[l] = at + __popc(same);
        __syncwarp();
    }
}

// zl::dynamic_header by the warp, which has llen and dlen: the number of
// entries that a run of equal lengths takes has a closed form, so every lane
// codes the runs that start at its symbols; the code-length code's own lengths
// are lane 0's. Every lane gets the result.
__device__ long long warp_dynamic_header(DeflateWarp &s, int lane)
{
    Codes &c = s.codes;
    auto &b = s.u.b;
    uint16_t *len16 = b.dep;  // the lengths, literals' then distances' (the code construction is done)
    int hl = kLitSyms, hd = kDistSyms;
    {
        int top = 256;
        for (int x = 257 + lane; x < kLitSyms; x += 32)
            if (c.llen[x]) top = x;
        hl = max(257, __reduce_max_sync(0xffffffffu, top) + 1);
        hd = max(1, __reduce_max_sync(0xffffffffu, lane < kDistSyms && c.dlen[lane] ? lane + 1 : 0));
    }
    const int n = hl + hd;
    for (int x = lane; x < n; x += 32) len16[x] = x < hl ? c.llen[x] : c.dlen[x - hl];
    if (lane < kClSyms) s.cnt[lane] = 0;
    __syncwarp();
    // run lengths: the next position where the length changes
    int out = 0;  // entries so far
    for (int x0 = 0; x0 < n; x0 += 32) {
        const int x = x0 + lane;
        const int v = x < n ? len16[x] : -1;
        const bool start = x < n && (x == 0 || len16[x - 1] != v);
        int run = 0, m = 0;
        if (start) {
            run = 1;
            while (x + run < n && len16[x + run] == v) ++run;
            // zeros: pieces of 138 (18), then 11-137 (18), 3-10 (17) or single
            // ones; others: one as it is, pieces of 6 (16), then 3-5 (16) or single
            const int rep = v ? run - 1 : run, q = v ? 6 : 138, rest = rep % q;
            m = (v ? 1 : 0) + rep / q + (rest >= 3 ? 1 : rest);
        }
        int inc = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (start) {
            int at = out + inc - m;
            auto put = [&](int e) {
                c.rle[at++] = (uint16_t)e;
                atomicAdd(&s.cnt[e & 31], 1u);
            };
            if (v) put(v);
            const int rep = v ? run - 1 : run, q = v ? 6 : 138, rest = rep % q;
            for (int k = 0; k < rep / q; ++k) put(v ? 16 | 3 << 8 : 18 | 127 << 8);
            if (v) {
                if (rest >= 3) put(16 | (rest - 3) << 8);
                else
                    for (int k = 0; k < rest; ++k) put(v);
            } else if (rest >= 11) {
                put(18 | (rest - 11) << 8);
            } else if (rest >= 3) {
                put(17 | (rest - 3) << 8);
            } else {
                for (int k = 0; k < rest; ++k) put(0);
            }
        }
        out += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncwarp();
    long long bits = -1;
    if (lane == 0) {
        c.hlit = hl;
        c.hdist = hd;
        c.nrle = out;
        bits = zl::code_length_code(c, s.cnt);
    }
    __syncwarp();
    int sum = 0;
    for (int i = lane; i < out; i += 32) {
        const int x = c.rle[i] & 31;
        sum += c.clen[x] + zl::rle_extra_bits(x);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    bits = __shfl_sync(0xffffffffu, bits, 0);
    return bits < 0 ? -1 : bits + sum;
}

// zl::data_bits (with the dynamic lengths) and zl::fixed_block_bits of the
// block's counts, summed by the warp instead of lane 0; the same integers.
__device__ void warp_block_bits(const DeflateWarp &s, const uint8_t *llen, const uint8_t *dlen, int lane,
                                long long &data, long long &fixed)
{
    long long a = 0, f = 0;
    for (int x = lane; x < zl::kLitSyms; x += 32) {
        const long long c = s.lf[x];
        a += c * llen[x];
        f += c * zl::fixed_lit_len(x);
    }
    if (lane < 29) {
        const long long c = s.lf[257 + lane];
        a += c * zl::len_extra(lane);
        f += c * zl::len_extra(lane);
    }
    if (lane < zl::kDistSyms) {
        const long long c = s.df[lane];
        a += c * (dlen[lane] + zl::dist_extra(lane));
        f += c * (5 + zl::dist_extra(lane));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        f += __shfl_xor_sync(0xffffffffu, f, o);
    }
    data = a;
    fixed = 3 + f;
}

// Serial bit writer of lane 0 into the ring (block headers).
struct RingW {
    uint32_t *ring;
    int bp;
    __device__ void put(unsigned long long v, int n)
    {
        const int sh = bp & 31, wi = bp >> 5;
        const unsigned long long lo = v << sh;
        ring[wi & kRingM] |= (uint32_t)lo;
        ring[(wi + 1) & kRingM] |= (uint32_t)(lo >> 32);
        if (sh && n + sh > 64) ring[(wi + 2) & kRingM] |= (uint32_t)(v >> (64 - sh));
        bp += n;
    }
};

__device__ __forceinline__ void ring_or(uint32_t *ring, int b, unsigned long long v)
{
    const int sh = b & 31, wi = b >> 5;
    const unsigned long long lo = v << sh;
    const uint32_t x0 = (uint32_t)lo, x1 = (uint32_t)(lo >> 32), x2 = sh ? (uint32_t)(v >> (64 - sh)) : 0u;
    if (x0) atomicOr(ring + (wi & kRingM), x0);
    if (x1) atomicOr(ring + ((wi + 1) & kRingM), x1);
    if (x2) atomicOr(ring + ((wi + 2) & kRingM), x2);
}

// The ring of one block's output: words [flushed, bp/32] are live; older
// words are in the output, their slots zero. Flushes keep a step of at most
// 32 items (48 bits each) clear of the live words. A first word that the
// block before shares (shared_word) goes to *head instead of the output.
struct Ring {
    uint32_t *ring, *dstw;
    int bp, flushed, wlimit, shared_word;
    uint32_t *head;
    __device__ void flush_to(int to, int lane)
    {
        for (int w = flushed + lane; w < to; w += 32) {
            if (w == shared_word) *head = ring[w & kRingM];
            else if (w < wlimit) dstw[w] = ring[w & kRingM];
            ring[w & kRingM] = 0;
        }
        flushed = to;
        __syncwarp();
    }
    __device__ void make_room(int lane, int words = 64)
    {
        if ((bp >> 5) + words >= flushed + kRingW) flush_to(bp >> 5, lane);
    }
};

// Sequence cursor: record index and the input position of its literals.
struct Cursor {
    int i, pos;
};

// Four bytes at any address as a little-endian word; reads whole aligned
// words (inputs carry tail room).
__device__ __forceinline__ uint32_t bytes4(const uint8_t *p)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    return __funnelshift_r(__ldg(w), __ldg(w + 1), 8 * (uint32_t)(a & 3));
}

// The codes of the first min(n, 4) bytes of w, one after the other.
__device__ __forceinline__ void pack4(const zl::Codes &cd, uint32_t w, int n, unsigned long long &v, int &bits)
{
    v = 0;
    bits = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t x = (w >> (8 * j)) & 0xffu;
        if (j < n) {
            v |= (unsigned long long)cd.lcode[x] << bits;
            bits += cd.llen[x];
        }
    }
}

// The items (literal bytes and match pieces) of the parse that start in
// [lo, hi), from cursor cur, 32 sequences per batch, one per lane. Literal
// runs of more than kShortLit bytes and matches of more than kShortPieces
// pieces are shared out over the warp, 128 bytes or 32 pieces a step; the
// other lanes take their own sequence whole, so that a batch costs one scan.
// MODE 0 counts symbols into s.lf/s.df; MODE 1 writes their codes into the
// ring; MODE 2 looks at no item. Returns the end of the bytes the items
// cover; `next` is set to the first sequence that reaches past that end.
constexpr int kShortLit = 32, kShortPieces = 4;
constexpr int kShortWords = 32 * (15 * kShortLit + 48 * kShortPieces) / 32 + 2;  // most ring words of a batch of short ones
static_assert(kShortWords + 1 < kRingW, "ring");

template <int MODE>
__device__ int block_items(DeflateWarp &s, const unsigned long long *seq, int nseq, Cursor cur, int lo, int hi,
                           const uint8_t *src, Ring *rg, Cursor *next, int lane)
{
    int cov = lo;
    int i0 = cur.i, pos = cur.pos;
    unsigned long long r = i0 + lane < nseq ? seq[i0 + lane] : 0ull;
    for (;;) {
        const int i = i0 + lane;
        const unsigned long long ahead = i + 32 < nseq ? seq[i + 32] : 0ull;  // the next batch
        const int lit = zl::seq_lit(r), m = zl::seq_mlen(r), d = zl::seq_dist(r);
        const int span = lit + m;
        int incl = span;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int ls = pos + incl - span, ms = ls + lit;
        const int span_total = __shfl_sync(0xffffffffu, incl, 31);
        // literal sub-range [a, b) and pieces [k0, k1) that start in [lo, hi)
        const int a = min(max(lo - ls, 0), lit), b = min(max(hi - ls, 0), lit);
        const int k0 = m ? zl::pieces_before(m, lo - ms) : 0, k1 = m ? zl::pieces_before(m, hi - ms) : 0;
        int nl = b - a, np = k1 - k0;
        int c = 0;
        if (np > 0) c = ms + zl::piece_start(m, k1 - 1) + zl::piece_len(m, k1 - 1);
        else if (nl > 0) c = ls + b;
        c = __reduce_max_sync(0xffffffffu, c);
        cov = max(cov, c);
        const uint8_t *lp = src + ls + a;
        if (MODE == 0) {
            // order does not matter: long ones by the warp, then every lane's own
            for (unsigned lng = __ballot_sync(0xffffffffu, nl > kShortLit); lng; lng &= lng - 1) {
                const int who = __ffs(lng) - 1;
                const int p0 = __shfl_sync(0xffffffffu, ls + a, who), n = __shfl_sync(0xffffffffu, nl, who);
#pragma unroll 2
                for (int k = 4 * lane; k < n; k += 128) {
                    const uint32_t w = bytes4(src + p0 + k);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (k + j < n) atomicAdd(&s.lf[(w >> (8 * j)) & 0xffu], 1u);
                }
            }
            for (unsigned lng = __ballot_sync(0xffffffffu, np > kShortPieces); lng; lng &= lng - 1) {
                const int who = __ffs(lng) - 1;
                const int mm = __shfl_sync(0xffffffffu, m, who), dd = __shfl_sync(0xffffffffu, d, who);
                const int e = __shfl_sync(0xffffffffu, k1, who);
                for (int k = __shfl_sync(0xffffffffu, k0, who) + lane; k < e; k += 32) {
                    atomicAdd(&s.lf[257 + zl::len_sym(zl::piece_len(mm, k))], 1u);
                    atomicAdd(&s.df[zl::dist_sym(dd)], 1u);
                }
            }
            if (nl <= kShortLit)
                for (int k = 0; k < nl; k += 4) {
                    const uint32_t w = bytes4(lp + k);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (k + j < nl) atomicAdd(&s.lf[(w >> (8 * j)) & 0xffu], 1u);
                }
            if (np > 0 && np <= kShortPieces) {
                for (int k = k0; k < k1; ++k) atomicAdd(&s.lf[257 + zl::len_sym(zl::piece_len(m, k))], 1u);
                atomicAdd(&s.df[zl::dist_sym(d)], (uint32_t)np);
            }
        } else if (MODE == 1) {
            const zl::Codes &cd = s.codes;
            // lanes [from, to) in turn: short ones together up to the next
            // long one, its literals or pieces, then on from there
            unsigned long_lit = __ballot_sync(0xffffffffu, nl > kShortLit);
            unsigned long_rep = __ballot_sync(0xffffffffu, np > kShortPieces);
            unsigned todo = __ballot_sync(0xffffffffu, nl + np > 0);
            while (todo) {
                const unsigned stops = (long_lit | long_rep) & todo;
                const int to = stops ? __ffs(stops) - 1 : 32;
                const unsigned below = to == 32 ? todo : todo & ((1u << to) - 1u);
                if (below) {
                    const bool mine = below >> lane & 1u;
                    // the first four literals and the first piece are
                    // looked up once (most sequences have no more)
                    unsigned long long v0 = 0, v1 = 0;
                    int n0 = 0, n1 = 0, bits = 0;
                    if (mine) {
                        if (nl > 0) pack4(cd, bytes4(lp), nl, v0, n0);
                        if (np > 0) n1 = zl::match_bits(cd, zl::piece_len(m, k0), d, v1);
                        bits = n0 + n1;
                        for (int k = 4; k < nl; k += 4) {
                            const uint32_t w = bytes4(lp + k);
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (k + j < nl) bits += cd.llen[(w >> (8 * j)) & 0xffu];
                        }
                        unsigned long long v;
                        for (int k = k0 + 1; k < k1; ++k) bits += zl::match_bits(cd, zl::piece_len(m, k), d, v);
                    }
                    int bi = bits;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, bi, o);
                        if (lane >= o) bi += t;
                    }
                    rg->make_room(lane, kShortWords);
                    if (mine) {
                        int at = rg->bp + bi - bits;
                        ring_or(rg->ring, at, v0);
                        at += n0;
                        for (int k = 4; k < nl; k += 4) {
                            unsigned long long v;
                            int n;
                            pack4(cd, bytes4(lp + k), nl - k, v, n);
                            ring_or(rg->ring, at, v);
                            at += n;
                        }
                        ring_or(rg->ring, at, v1);
                        at += n1;
                        for (int k = k0 + 1; k < k1; ++k) {
                            unsigned long long v;
                            const int n = zl::match_bits(cd, zl::piece_len(m, k), d, v);
                            ring_or(rg->ring, at, v);
                            at += n;
                        }
                    }
                    rg->bp += __shfl_sync(0xffffffffu, bi, 31);
                    __syncwarp();  // the next flush reads these words
                    todo &= ~below;
                }
                if (to == 32) continue;
                if (long_lit >> to & 1u) {
                    const int p0 = __shfl_sync(0xffffffffu, ls + a, to), n = __shfl_sync(0xffffffffu, nl, to);
                    for (int t0 = 0; t0 < n; t0 += 128) {
                        const int k = t0 + 4 * lane;
                        const uint32_t w = k < n ? bytes4(src + p0 + k) : 0u;
                        unsigned long long v;
                        int nb;
                        pack4(cd, w, n - k, v, nb);
                        int bi = nb;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int t = __shfl_up_sync(0xffffffffu, bi, o);
                            if (lane >= o) bi += t;
                        }
                        rg->make_room(lane, 64);
                        if (nb) ring_or(rg->ring, rg->bp + bi - nb, v);
                        rg->bp += __shfl_sync(0xffffffffu, bi, 31);
                        __syncwarp();
                    }
                    long_lit &= ~(1u << to);
                    if (lane == to) nl = 0;
                    // its match: with the next short ones, or below
                }
                if (long_rep >> to & 1u) {
                    // the literals before it are written (a short run first)
                    const int n = __shfl_sync(0xffffffffu, nl, to);
                    if (n > 0) {
                        const int p0 = __shfl_sync(0xffffffffu, ls + a, to);
                        const uint32_t x = lane < n ? src[p0 + lane] : 0u;
                        const int nb = lane < n ? cd.llen[x] : 0;
                        int bi = nb;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int t = __shfl_up_sync(0xffffffffu, bi, o);
                            if (lane >= o) bi += t;
                        }
                        rg->make_room(lane, 64);
                        if (nb) ring_or(rg->ring, rg->bp + bi - nb, cd.lcode[x]);
                        rg->bp += __shfl_sync(0xffffffffu, bi, 31);
                        __syncwarp();
                    }
                    const int mm = __shfl_sync(0xffffffffu, m, to), dd = __shfl_sync(0xffffffffu, d, to);
                    const int e = __shfl_sync(0xffffffffu, k1, to);
                    for (int t0 = __shfl_sync(0xffffffffu, k0, to); t0 < e; t0 += 32) {
                        unsigned long long v = 0;
                        const int k = t0 + lane, nb = k < e ? zl::match_bits(cd, zl::piece_len(mm, k), dd, v) : 0;
                        int bi = nb;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int t = __shfl_up_sync(0xffffffffu, bi, o);
                            if (lane >= o) bi += t;
                        }
                        rg->make_room(lane, 64);
                        if (nb) ring_or(rg->ring, rg->bp + bi - nb, v);
                        rg->bp += __shfl_sync(0xffffffffu, bi, 31);
                        __syncwarp();
                    }
                    long_rep &= ~(1u << to);
                    todo &= ~(1u << to);
                }
            }
        }
        __syncwarp();
        const bool last = pos + span_total >= hi || i0 + 32 >= nseq;
        if (last) {
            // the next block starts at the first sequence reaching past cov
            const unsigned beyond = __ballot_sync(0xffffffffu, i < nseq && ls + span > cov);
            if (beyond) {
                const int f = __ffs(beyond) - 1;
                next->i = i0 + f;
                next->pos = __shfl_sync(0xffffffffu, ls, f);
            } else {
                next->i = min(i0 + 32, nseq);
                next->pos = pos + span_total;
            }
            return cov;
        }
        pos += span_total;
        i0 += 32;
        r = ahead;
    }
}

// Validation of a chunk's parse: lengths sum to L, matches of at least 3
// bytes within the window and the output so far.
__device__ bool parse_ok(const unsigned long long *seq, int nseq, int L, int lane)
{
    int pos = 0;
    bool ok = true;
    constexpr int kA = 8;  // batches loaded ahead
    unsigned long long q[kA];
#pragma unroll
    for (int u = 0; u < kA; ++u) q[u] = 32 * u + lane < nseq ? seq[32 * u + lane] : 0ull;
    for (int i0 = 0; i0 < nseq; i0 += 32) {
        const unsigned long long r = q[0];
#pragma unroll
        for (int u = 0; u + 1 < kA; ++u) q[u] = q[u + 1];
        q[kA - 1] = i0 + 32 * kA + lane < nseq ? seq[i0 + 32 * kA + lane] : 0ull;
        const int lit = zl::seq_lit(r), m = zl::seq_mlen(r), d = zl::seq_dist(r);
        int incl = lit + m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        const int ms = pos + incl - m;
        ok = ok && (m == 0 || (m >= 3 && d >= 1 && d <= zl::kMaxDist && d <= ms));
        pos += __shfl_sync(0xffffffffu, incl, 31);
        if (pos > L) ok = false;
    }
    return __all_sync(0xffffffffu, ok) && pos == L;
}

// One CTA per chunk. A chunk's DEFLATE blocks (five per block record) depend
// on one another only through where they start in the input (a match may reach
// past a block's end) and in the output: warp 0 finds the former from the
// parse alone for the next kZWarps blocks, every warp then counts one block's
// symbols and builds its codes, one thread picks the codings and adds up the
// bits, and every warp writes its block at its place. The word two blocks
// share is put together at the end. With a warp per chunk doing the blocks in
// turn, 512 chunks (256^3) left three warps to an SM: the
// DEFLATE stage took 3.0 ms, with a CTA each 0.8 ms.
struct DeflateBlock {
    int lo, hi, cov;
    Cursor cur;
    long long dyn, fix;  // bits of the dynamic coding (-1: none) and of the fixed one
    int mode, start, bits;
    uint32_t head, tail;  // its bits of a first and a last word that it shares
};

__global__ void __launch_bounds__(kZWarps * 32, 4)
deflate_kernel(const uint8_t *__restrict__ in, const long long *in_off, const int *in_len,
               const uint8_t *__restrict__ sq, const long long *seq_off, const int *seq_bytes, int nchunks,
               int records, uint8_t *__restrict__ out, long long out_slot, long long *out_off, int *out_len)
{
    extern __shared__ __align__(16) unsigned char deflate_smem[];
    DeflateWarp *sw = reinterpret_cast<DeflateWarp *>(deflate_smem);
    __shared__ DeflateBlock blk[kZWarps];
    __shared__ int s_n, s_ok, s_err;
    __shared__ unsigned long long s_sum[kZWarps][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    DeflateWarp &s = sw[warp];
    for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint8_t *src = in + in_off[c];
        const int L = in_len[c];
        const int sb = seq_bytes[c];
        const unsigned long long *seq = reinterpret_cast<const unsigned long long *>(sq + seq_off[c]);
        const int nseq = sb >= 8 && (sb & 7) == 0 ? sb / 8 : 0;
        uint8_t *dst = out + (long long)c * out_slot;
        uint32_t *dstw = reinterpret_cast<uint32_t *>(dst);
        const int wlimit = (int)(out_slot / 4);
        if (threadIdx.x == 0) {
            out_off[c] = (long long)c * out_slot;
            s_err = 0;
        }
        if (warp == 0) {
            const bool ok = nseq > 0 && parse_ok(seq, nseq, L, lane);
            if (lane == 0) s_ok = ok;
        } else {
            // Adler-32 of the input (chunks start on 4-byte boundaries)
            unsigned long long sa, sbs;
            adler_sums<false>(src, L, threadIdx.x - 32, 32 * (kZWarps - 1), sa, sbs);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sa += __shfl_xor_sync(0xffffffffu, sa, o);
                sbs += __shfl_xor_sync(0xffffffffu, sbs, o);
            }
            if (lane == 0) {
                s_sum[warp][0] = sa;
                s_sum[warp][1] = sbs;
            }
        }
        __syncthreads();
        if (!s_ok) {
            if (threadIdx.x == 0) out_len[c] = -1;
            __syncthreads();
            continue;
        }
        zl::Bounds bnd;  // warp 0's
        bnd.init(src, L, records != 0);
        Cursor cur{0, 0};
        int lo = 0, nblk = 0;
        int bp = 16;               // thread 0's: bits written, and those of the last, partial word
        uint32_t carry = 0x9c78u;  // (the zlib header at first)
        bool final = false;
        while (!final) {
            // ---- the next blocks
            if (warp == 0) {
                int n = 0, err = 0;
                bool end = false;
                while (n < kZWarps && !end) {
                    const int hi = bnd.next(lo);
                    Cursor nxt;
                    const int cov = block_items<2>(s, seq, nseq, cur, lo, hi, src, nullptr, &nxt, lane);
                    if (lane == 0) {
                        blk[n].lo = lo;
                        blk[n].hi = hi;
                        blk[n].cov = cov;
                        blk[n].cur = cur;
                    }
                    ++n;
                    end = cov >= L;
                    if (!end && cov <= lo) err = 3;             // every block makes progress
                    if (++nblk > L / zl::kMinBlock + 2) err = 4;
                    if (err) break;
                    cur = nxt;
                    lo = cov;
                }
                if (lane == 0) {
                    s_n = n;
                    if (err) s_err = err;
                }
            }
            __syncthreads();
            const int n = s_n;
            if (s_err) break;
            final = blk[n - 1].cov >= L;
            DeflateBlock &b = blk[warp];
            // ---- symbol counts of the items starting in [lo, hi), codes, sizes
            if (warp < n) {
                for (int x = lane; x < 288; x += 32) s.lf[x] = x == 256 ? 1u : 0u;
                s.df[lane] = 0;
                __syncwarp();
                Cursor nxt;
                block_items<0>(s, seq, nseq, b.cur, b.lo, b.hi, src, nullptr, &nxt, lane);
                bool ok = warp_code(s, s.lf, zl::kLitSyms, s.codes.llen, lane);
                ok = warp_code(s, s.df, zl::kDistSyms, s.codes.dlen, lane) && ok;
                long long dbits, fbits;
                warp_block_bits(s, s.codes.llen, s.codes.dlen, lane, dbits, fbits);
                Codes &cd = s.codes;
                if (lane < 288 - zl::kLitSyms) cd.llen[zl::kLitSyms + lane] = 0;
                if (lane < 32 - zl::kDistSyms) cd.dlen[zl::kDistSyms + lane] = 0;
                __syncwarp();
                if (ok) {
                    warp_canon_codes(s, cd.llen, 288, cd.lcode, lane);
                    warp_canon_codes(s, cd.dlen, 32, cd.dcode, lane);
                }
                const long long hb = ok ? warp_dynamic_header(s, lane) : -1;
                if (lane == 0) {
                    b.dyn = hb >= 0 ? hb + dbits : -1;
                    b.fix = fbits;
                }
            }
            __syncthreads();
            // ---- every block's coding, the one with the fewest bits, and place
            if (threadIdx.x == 0) {
                int at = bp;
                for (int w = 0; w < n; ++w) {
                    DeflateBlock &q = blk[w];
                    const long long sto =
                        q.cov - q.lo <= zl::kStoredMax ? zl::stored_block_bits(at, q.cov - q.lo) : -1;
                    int mode = 2;
                    long long best = q.dyn;
                    if (q.dyn < 0 || q.fix <= q.dyn) {
                        mode = 1;
                        best = q.fix;
                    }
                    if (sto >= 0 && sto <= best) {
                        mode = 0;
                        best = sto;
                    }
                    q.mode = mode;
                    q.start = at;
                    q.bits = (int)best;
                    q.head = q.tail = 0;
                    at += (int)best;
                }
            }
            __syncthreads();
            // ---- the blocks
            if (warp < n) {
                const bool last = b.cov >= L;
                for (int w = lane; w < kRingW; w += 32) s.u.ring[w] = 0;
                if (b.mode == 1 && lane == 0) zl::fixed_codes(s.codes);
                __syncwarp();
                Ring rg{s.u.ring, dstw, b.start, b.start >> 5, wlimit, b.start & 31 ? b.start >> 5 : -1, &b.head};
                RingW wr{s.u.ring, rg.bp};
                if (lane == 0) {
                    if (b.mode == 0) {
                        wr.put(last ? 1u : 0u, 3);
                        wr.bp = (wr.bp + 7) & ~7;
                        const unsigned m = (unsigned)(b.cov - b.lo);
                        wr.put(m | (~m & 0xffffu) << 16, 32);
                    } else if (b.mode == 1) {
                        wr.put((last ? 1u : 0u) | 1u << 1, 3);
                    } else {
                        zl::put_dynamic_header(wr, s.codes, last);
                    }
                }
                __syncwarp();
                rg.bp = __shfl_sync(0xffffffffu, wr.bp, 0);
                if (b.mode == 0) {
                    // bytes to the word boundary, whole words, the last bytes
                    const int m = b.cov - b.lo, h = min(m, (32 - (rg.bp & 31)) / 8 & 3), nw = (m - h) >> 2;
                    const uint8_t *q = src + b.lo;
                    if (lane < h) ring_or(rg.ring, rg.bp + 8 * lane, q[lane]);
                    rg.bp += 8 * h;
                    __syncwarp();
                    if (nw > 0) {  // at a word boundary
                        rg.flush_to(rg.bp >> 5, lane);
                        const uintptr_t a = reinterpret_cast<uintptr_t>(q + h);
                        const uint32_t *sw32 = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
                        const uint32_t sh = 8 * (uint32_t)(a & 3);
                        const int w0 = rg.bp >> 5;
#pragma unroll 4
                        for (int i = lane; i < nw; i += 32)
                            if (w0 + i < wlimit)
                                dstw[w0 + i] = sh ? __funnelshift_r(sw32[i], sw32[i + 1], sh) : sw32[i];
                        rg.bp += 32 * nw;
                        rg.flushed = rg.bp >> 5;
                    }
                    const int t = m - h - 4 * nw;
                    if (lane < t) ring_or(rg.ring, rg.bp + 8 * lane, q[h + 4 * nw + lane]);
                    rg.bp += 8 * t;
                    __syncwarp();
                } else {
                    Cursor dummy;
                    block_items<1>(s, seq, nseq, b.cur, b.lo, b.hi, src, &rg, &dummy, lane);
                    rg.make_room(lane);
                    if (lane == 0) ring_or(rg.ring, rg.bp, s.codes.lcode[256]);
                    rg.bp += s.codes.llen[256];
                    __syncwarp();
                }
                rg.flush_to(rg.bp >> 5, lane);
                if (lane == 0) {
                    b.tail = rg.bp & 31 ? s.u.ring[(rg.bp >> 5) & kRingM] : 0u;
                    if (rg.bp - b.start != b.bits) s_err = 2;  // written bits must be the counted ones
                }
            }
            __syncthreads();
            if (s_err) break;
            // ---- the words that blocks share
            if (threadIdx.x == 0) {
                for (int w = 0; w < n; ++w) {
                    const DeflateBlock &q = blk[w];
                    const int e = q.start + q.bits;
                    if (e >> 5 == q.start >> 5) {
                        carry |= q.tail;
                    } else {
                        if (q.start & 31 && q.start >> 5 < wlimit) dstw[q.start >> 5] = carry | q.head;
                        carry = q.tail;
                    }
                    bp = e;
                }
            }
            __syncthreads();  // blk is free
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int nbytes = (bp + 7) >> 3;
            if (s_err || nbytes + 4 > out_slot) {
                out_len[c] = -2;
            } else {
                if (bp & 31) dstw[bp >> 5] = carry;
                unsigned long long sa = 0, sbs = 0;
                for (int w = 1; w < kZWarps; ++w) {
                    sa += s_sum[w][0];
                    sbs += s_sum[w][1];
                }
                const unsigned adler = adler_of(sa, sbs, L);
                dst[nbytes] = (uint8_t)(adler >> 24);
                dst[nbytes + 1] = (uint8_t)(adler >> 16);
                dst[nbytes + 2] = (uint8_t)(adler >> 8);
                dst[nbytes + 3] = (uint8_t)adler;
                out_len[c] = nbytes + 4;
            }
        }
        __syncthreads();
    }
}

}  // namespace cz

using namespace cz;

cudaError_t cz_launch_deflate(const uint8_t *in, const long long *in_off, const int *in_len, const uint8_t *seq,
                              const long long *seq_off, const int *seq_bytes, int nchunks, int records, uint8_t *out,
                              long long out_slot, long long *out_off, int *out_len, int grid, cudaStream_t st)
{
    if (nchunks <= 0) return cudaSuccess;
    const int sm = (int)sizeof(DeflateWarp) * kZWarps;
    const cudaError_t e = cudaFuncSetAttribute(deflate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    deflate_kernel<<<grid, kZWarps * 32, sm, st>>>(in, in_off, in_len, seq, seq_off, seq_bytes, nchunks, records, out,
                                                   out_slot, out_off, out_len);
    return cudaGetLastError();
}

cudaError_t cz_launch_inflate(const uint8_t *in, const long long *in_off, const int *in_len, int nchunks, uint8_t *out,
                              const long long *out_off, const int *out_cap, int *out_len, int grid, cudaStream_t st,
                              long long cap)
{
    if (nchunks <= 0) return cudaSuccess;
    inflate_kernel<<<grid, 64, 0, st>>>(in, in_off, in_len, nchunks, out, out_off, out_cap, out_len, cap);
    return cudaGetLastError();
}
