// cz_inflate.cuh -- the serial part of zlib decoding (RFC 1950 wrapper, RFC
// 1951 DEFLATE), shared by the GPU kernel (run by one lane per chunk) and the
// host test harness: bit reader, canonical Huffman codes, and the decoder
// state machine that writes literals and records matches in batches.
//
// The length and distance tables of RFC 1951 3.2.5 are computed from their
// closed forms; the code-length code order of 3.2.7 is packed in constants.
#pragma once
#include <stdint.h>

#include "cz_arith.cuh"  // CZ_HD

// member functions (CZ_HD is `static inline` in host builds)
#if defined(__CUDACC__)
#define CZ_MEM __host__ __device__ __forceinline__
#else
#define CZ_MEM inline
#endif

namespace cz {
namespace zl {

constexpr int kMaxBits = 15;
constexpr int kFastBits = 10;  // codes up to this length decode with one table lookup
constexpr int kFastMask = (1 << kFastBits) - 1;
constexpr int kClBits = 7;     // code-length codes

// RFC 1951 3.2.5: length codes 257..285 (li = code - 257), distance codes 0..29
CZ_HD int len_extra(int li) { return li < 8 || li == 28 ? 0 : (li - 4) >> 2; }
CZ_HD int len_base(int li)
{
    if (li < 8) return 3 + li;
    if (li == 28) return 258;
    return (((li - 8) & 3) + 4 << len_extra(li)) + 3;
}
CZ_HD int dist_extra(int ds) { return ds < 4 ? 0 : (ds - 2) >> 1; }
CZ_HD int dist_base(int ds) { return ds < 4 ? ds + 1 : ((2 + (ds & 1)) << dist_extra(ds)) + 1; }
// RFC 1951 3.2.7: 16,17,18,0,8,7,9,6,10,5,11,4,12,3,13,2,14,1,15 (5 bits each)
CZ_HD int cl_order(int i)
{
    const unsigned long long lo = 16ull | 17ull << 5 | 18ull << 10 | 0ull << 15 | 8ull << 20 | 7ull << 25 |
                                  9ull << 30 | 6ull << 35 | 10ull << 40 | 5ull << 45 | 11ull << 50 | 4ull << 55;
    const unsigned long long hi = 12ull | 3ull << 5 | 13ull << 10 | 2ull << 15 | 14ull << 20 | 1ull << 25 | 15ull << 30;
    return i < 12 ? (int)((lo >> (5 * i)) & 31) : (int)((hi >> (5 * (i - 12))) & 31);
}

// Bit reader over 32-bit words: cnt unread bits in (lo, hi), the next word
// already loaded. The GPU reads aligned words, so `skip` bits of the first
// one precede the input. Past the input the last word repeats: over() tells
// when such bits were consumed. No branches: on the GPU a single lane runs
// this, and every branch costs it a dozen cycles.
struct Bits {
    const uint8_t *p;  // the words
    int last, wi;      // last word that holds input, the next one to take
    int skip, cnt;
    long long limit;   // input bits, skip included
    uint32_t lo, hi, nw;
    CZ_MEM uint32_t word(int i) const
    {
        const int k = i < last ? i : last;
#if defined(__CUDA_ARCH__)
        return __ldg(reinterpret_cast<const uint32_t *>(p) + k);
#else
        uint32_t w = 0;
        const long long left = limit / 8 - 4ll * k;
        memcpy(&w, p + 4ll * k, (size_t)(left < 4 ? left : 4));
        return w;
#endif
    }
    CZ_MEM void init(const uint8_t *src, long long n)  // n > 0
    {
#if defined(__CUDA_ARCH__)
        skip = 8 * (int)(reinterpret_cast<uintptr_t>(src) & 3);
#else
        skip = 0;
#endif
        p = src - skip / 8;
        limit = 8 * n + skip;
        last = (int)((limit + 31) / 32) - 1;
        seek(0);
    }
    // to input byte `at`
    CZ_MEM void seek(long long at)
    {
        const long long bit = 8 * at + skip;
        wi = (int)(bit >> 5);
        const int r = (int)(bit & 31);
        lo = word(wi) >> r;
        hi = 0;
        cnt = 32 - r;
        ++wi;
        nw = word(wi);
    }
    // at least 33 bits
    CZ_MEM void refill()
    {
#if defined(__CUDA_ARCH__)
        const bool need = cnt <= 32;
        lo |= __funnelshift_lc(0u, nw, cnt);                   // nw << cnt, 0 from 32 on
        hi = need ? __funnelshift_lc(nw, 0u, cnt) : hi;        // nw >> (32 - cnt)
        cnt += need ? 32 : 0;
        wi += need ? 1 : 0;
        nw = word(wi);
#else
        if (cnt > 32) return;
        lo |= cnt < 32 ? nw << cnt : 0u;
        hi = cnt ? nw >> (32 - cnt) : 0u;
        cnt += 32;
        ++wi;
        nw = word(wi);
#endif
    }
    CZ_MEM void drop(int n)  // n < 32
    {
#if defined(__CUDA_ARCH__)
        lo = __funnelshift_r(lo, hi, n);
#else
        lo = n ? lo >> n | hi << (32 - n) : lo;
#endif
        hi >>= n;
        cnt -= n;
    }
    CZ_MEM unsigned get(int n)  // n < 32
    {
        refill();
        const unsigned v = lo & ((1u << n) - 1u);
        drop(n);
        return v;
    }
    CZ_MEM void align()
    {
        const int n = cnt & 7;
        drop(n);
    }
    CZ_MEM long long bit() const { return 32ll * wi - cnt; }
    CZ_MEM bool over() const { return bit() > limit; }  // bits past the end were consumed
    CZ_MEM long long byte() const { return (bit() - skip) >> 3; }       // when aligned
    CZ_MEM long long size() const { return (limit - skip) >> 3; }
};

// Canonical code: count[len] codes of each length, symbols sorted by code,
// and a table indexed by the next kFastBits input bits. Entries of the
// literal/length code:
//   literals: bits 0-4 the bits of their codes, 8-15 and 16-23 their values,
//     24-27 the first one's code length, 28-29 how many (1 or 2);
//   a length: bits 0-7 zero (nothing is consumed by looking it up, so further
//     lookups meet it again), 8-16 its base (0: end of block), 17-19 its extra
//     bits, 24-27 its code length, 31 set;
//   0: a longer code, or none.
// Entries of the distance code: bits 0-3 bits to consume (0: a longer code or
// none), 4-7 extra bits, 8-22 base.
// lim and shift decode any length: the length is the smallest l whose codes
// end above the next kMaxBits bits (first bit highest; canonical codes grow
// with length), the symbol sym[code + shift[l]].
struct Huff {
    unsigned short count[kMaxBits + 1];
    unsigned short sym[288];
    unsigned short lim[kMaxBits + 1];
    short shift[kMaxBits + 1];
    unsigned int fast[1 << kFastBits];
};
// The next kMaxBits bits with the first one highest.
CZ_HD unsigned rev_bits(unsigned v)
{
#if defined(__CUDA_ARCH__)
    return __brev(v) >> (32 - kMaxBits);
#else
    unsigned r = 0;
    for (int k = 0; k < kMaxBits; ++k) r |= ((v >> k) & 1u) << (kMaxBits - 1 - k);
    return r;
#endif
}
// Symbol of the code at the low bits of v and its length; -1: no code.
CZ_HD int long_code(const Huff &h, unsigned v, int &len)
{
    const unsigned r = rev_bits(v);
    int l = 1;
    while (l <= kMaxBits && r >= h.lim[l]) ++l;
    len = l;
    return l <= kMaxBits ? h.sym[(int)(r >> (kMaxBits - l)) + h.shift[l]] : -1;
}

CZ_HD int literals(unsigned e) { return (int)((e >> 28) & 3u); }
CZ_HD unsigned lit_entry(int sym, int len)
{
    const unsigned l = (unsigned)len;
    if (sym < 256) return l | (unsigned)sym << 8 | l << 24 | 1u << 28;
    if (sym == 256) return l << 24 | 1u << 31;
    const int li = sym - 257;
    return li < 29 ? (unsigned)len_base(li) << 8 | (unsigned)len_extra(li) << 17 | l << 24 | 1u << 31 : 0u;
}
CZ_HD unsigned dist_entry(int sym, int len)
{
    return sym < 30 ? (unsigned)len | (unsigned)dist_extra(sym) << 4 | (unsigned)dist_base(sym) << 8 : 0u;
}
// Entry i with the literal that follows it added where both codes fit.
CZ_HD unsigned pair_entry(const unsigned *fast, int i)
{
    const unsigned e = fast[i];
    if (!literals(e)) return e;
    const unsigned l1 = (e >> 24) & 15u, f = fast[i >> l1], l2 = (f >> 24) & 15u;
    if (!literals(f) || l1 + l2 > (unsigned)kFastBits) return e;
    return (l1 + l2) | (e & 0xff00u) | (f & 0xff00u) << 8 | l1 << 24 | 2u << 28;
}
// Whether a set of lengths is one that zlib takes: not oversubscribed, and
// complete unless it is empty or a single code of length 1 (the code-length
// code must be complete).
CZ_HD bool lengths_ok(const unsigned short *count, bool codelen)
{
    int left = 1, maxlen = 0;
    for (int i = 1; i <= kMaxBits; ++i) {
        left <<= 1;
        left -= count[i];
        if (left < 0) return false;
        if (count[i]) maxlen = i;
    }
    return !(left > 0 && maxlen > 0 && (codelen || maxlen != 1));
}

// Builds the code from lengths (serially; the GPU kernel has its own, by the
// warp). False for a set that zlib rejects.
CZ_HD bool build(Huff &h, const unsigned char *len, int n, bool lit)
{
    for (int i = 0; i <= kMaxBits; ++i) h.count[i] = 0;
    for (int s = 0; s < n; ++s) h.count[len[s]]++;
    h.count[0] = 0;
    if (!lengths_ok(h.count, false)) return false;
    unsigned short offs[kMaxBits + 1];
    offs[1] = 0;
    for (int i = 1; i < kMaxBits; ++i) offs[i + 1] = offs[i] + h.count[i];
    for (int l = 1, first = 0; l <= kMaxBits; ++l) {
        first = (first + (l > 1 ? h.count[l - 1] : 0)) << 1;
        h.lim[l] = (unsigned short)((first + h.count[l]) << (kMaxBits - l));
        h.shift[l] = (short)(offs[l] - first);
    }
    for (int s = 0; s < n; ++s)
        if (len[s]) h.sym[offs[len[s]]++] = (unsigned short)s;
    // lookup table: canonical codes in symbol order per length, bit-reversed
    // (the stream sends codes most significant bit first)
    for (int i = 0; i <= kFastMask; ++i) h.fast[i] = 0;
    int next[kFastBits + 1], code = 0;
    next[0] = 0;
    for (int l = 1; l <= kFastBits; ++l) {
        code = (code + h.count[l - 1]) << 1;
        next[l] = code;
    }
    for (int s = 0; s < n; ++s) {
        const int l = len[s];
        if (!l || l > kFastBits) continue;
        unsigned v = (unsigned)next[l]++, r = 0;
        for (int k = 0; k < l; ++k) {
            r = (r << 1) | (v & 1u);
            v >>= 1;
        }
        const unsigned e = lit ? lit_entry(s, l) : dist_entry(s, l);
        for (unsigned i = r; i <= (unsigned)kFastMask; i += 1u << l) h.fast[i] = e;
    }
    if (lit)
        for (int i = 0; i <= kFastMask; ++i) h.fast[i] = pair_entry(h.fast, i);
    return true;
}

// The code-length code's table (kClBits bits): length << 5 | symbol, 0 none.
CZ_HD bool build_cl(unsigned *fast, const unsigned char *len)
{
    unsigned short count[kMaxBits + 1];
    for (int i = 0; i <= kMaxBits; ++i) count[i] = 0;
    for (int s = 0; s < 19; ++s) count[len[s]]++;
    count[0] = 0;
    if (!lengths_ok(count, true)) return false;
    for (int i = 0; i < 1 << kClBits; ++i) fast[i] = 0;
    int code = 0;
    for (int l = 1; l <= kClBits; ++l) {
        code <<= 1;
        for (int s = 0; s < 19; ++s) {
            if (len[s] != l) continue;
            unsigned v = (unsigned)code++, r = 0;
            for (int k = 0; k < l; ++k) {
                r = (r << 1) | (v & 1u);
                v >>= 1;
            }
            for (unsigned i = r; i < 1u << kClBits; i += 1u << l) fast[i] = (unsigned)(l << 5 | s);
        }
    }
    return true;
}

// A few symbols: the literals of three table entries in order, then m: 0
// nothing, bit 31 set: a literal in the low byte, else a match, length |
// distance << 9.
struct Record {
    unsigned e[3], m;
};

// Decoder state.
struct Inflater {
    Bits b;
    long long op;  // output of step() so far (literals, recorded matches and runs)
    int err, final_block, in_block, btype;
    int nlen, ndist;  // a Huffman block's code lengths
    long long stored_left;
    // a stored block's bytes, for the caller to copy: input position, output
    // position (by step()), length (run_n = 0: none)
    long long run_src, run_dst, run_n;

    // Reads the zlib header; err != 0 if it is not a deflate stream without
    // a preset dictionary (RFC 1950 2.2).
    CZ_MEM void start(const uint8_t *src, long long n)
    {
        op = 0;
        err = final_block = in_block = btype = 0;
        nlen = ndist = 0;
        stored_left = 0;
        run_src = run_dst = run_n = 0;
        if (n <= 0) {
            err = 1;
            return;
        }
        b.init(src, n);
        const unsigned cmf = b.get(8), flg = b.get(8);
        if (b.over() || (cmf & 15) != 8 || (cmf >> 4) > 7 || ((cmf << 8) | flg) % 31 || (flg & 32)) err = 1;
    }

    // Reads a block header at the current position (BFINAL, BTYPE; LEN/NLEN
    // of a stored block; the code lengths of a Huffman block into lens).
    // Returns err (0: the block's data follows). scratch: 1 << kClBits words.
    CZ_MEM int block_header(unsigned *scratch, unsigned char *lens)
    {
        final_block = (int)b.get(1);
        btype = (int)b.get(2);
        in_block = 1;
        if (btype == 0) {
            b.align();
            const unsigned l = b.get(16), nl = b.get(16);
            if ((l ^ 0xffffu) != nl || b.over()) return err = 2;
            stored_left = l;
        } else if (btype == 1) {
            for (int i = 0; i < 288; ++i) lens[i] = i < 144 ? 8 : (i < 256 ? 9 : (i < 280 ? 7 : 8));
            // all 32 fixed distance codes (30 and 31 never occur, RFC 1951 3.2.6)
            for (int i = 0; i < 32; ++i) lens[288 + i] = 5;
            nlen = 288;
            ndist = 32;
        } else if (btype == 2) {
            nlen = (int)b.get(5) + 257;
            ndist = (int)b.get(5) + 1;
            const int ncode = (int)b.get(4) + 4;
            if (nlen > 286 || ndist > 30) return err = 3;
            for (int i = 0; i < 19; ++i) lens[i] = 0;
            for (int i = 0; i < ncode; ++i) lens[cl_order(i)] = (unsigned char)b.get(3);
            if (!build_cl(scratch, lens)) return err = 4;
            int i = 0, prev = 0;
            while (i < nlen + ndist) {
                b.refill();
                const unsigned e = scratch[b.lo & ((1u << kClBits) - 1)];
                if (!e) return err = 5;
                b.drop((int)(e >> 5));
                const int sym = (int)(e & 31u);
                if (b.over()) return err = 5;
                if (sym < 16) {
                    lens[i++] = (unsigned char)sym;
                    prev = sym;
                    continue;
                }
                int rep = 0, val = 0;
                if (sym == 16) {
                    if (i == 0) return err = 6;
                    val = prev;
                    rep = 3 + (int)b.get(2);
                } else if (sym == 17) {
                    rep = 3 + (int)b.get(3);
                } else {
                    rep = 11 + (int)b.get(7);
                }
                prev = val;
                if (i + rep > nlen + ndist) return err = 7;
                while (rep--) lens[i++] = (unsigned char)val;
            }
            if (lens[256] == 0) return err = 8;
        } else {
            return err = 11;
        }
        return 0;
    }

    // A stored block's data as a run; false (err) if the input ends first.
    CZ_MEM bool stored_run()
    {
        const long long from = b.byte();  // the block's data is byte aligned
        if (from + stored_left > b.size()) {
            err = 13;
            return false;
        }
        run_src = from;
        run_n = stored_left;
        b.seek(from + stored_left);
        in_block = 0;
        return true;
    }

    // The next record of a Huffman block; in_block = 0 at its end; err for a
    // code that does not exist. Bits consumed past the input are for the
    // caller to notice (b.over()). What bounds a chunk on the GPU is this
    // function's instructions, one after the other in a single lane: three
    // lookups in a row without a branch (an entry's low bits are the shift to
    // the next, the low bytes' sum what they consume), then, unless the third
    // is a literal, a match decoded as if its codes were in the tables, and one
    // branch for everything rare.
    CZ_MEM Record record(const Huff &lit, const Huff &dist)
    {
        const char *tab = reinterpret_cast<const char *>(lit.fast);
        constexpr unsigned kAt = (unsigned)kFastMask << 2;  // index as a byte offset
        Record r;
        b.refill();
        unsigned w = b.lo << 2;
        r.e[0] = *reinterpret_cast<const unsigned *>(tab + (w & kAt));
        w >>= r.e[0] & 31u;
        r.e[1] = *reinterpret_cast<const unsigned *>(tab + (w & kAt));
        w >>= r.e[1] & 31u;
        r.e[2] = *reinterpret_cast<const unsigned *>(tab + (w & kAt));
        r.m = 0;
        b.drop((int)((r.e[0] + r.e[1] + r.e[2]) & 31u));
        const unsigned e2 = r.e[2];
        if (literals(e2) == 0) {
            b.refill();
            const Bits save = b;
            int base = (int)((e2 >> 8) & 511u);
            const int x = (int)((e2 >> 17) & 7u);
            b.drop((int)((e2 >> 24) & 15u));
            const unsigned len = (unsigned)base + (b.lo & ((1u << x) - 1u));
            b.drop(x);
            b.refill();
            const unsigned d = dist.fast[b.lo & kFastMask];
            const int ld = (int)(d & 15u), xd = (int)((d >> 4) & 15u);
            b.drop(ld);
            r.m = len | ((d >> 8) + (b.lo & ((1u << xd) - 1u))) << 9;
            b.drop(xd);
            if (base == 0 || ld == 0) {
                b = save;
                r.m = rare(e2, lit, dist);
            }
        }
        return r;
    }
    // Its rare ends: the end of the block, codes longer than the tables'.
    CZ_MEM unsigned rare(unsigned e2, const Huff &lit, const Huff &dist)
    {
        int base = (int)((e2 >> 8) & 511u), x = (int)((e2 >> 17) & 7u), lc = (int)((e2 >> 24) & 15u);
        if (e2 == 0u) {
            const int sym = long_code(lit, b.lo, lc);
            if (sym < 0 || sym > 285) {
                err = sym < 0 ? 14 : 16;
                return 0u;
            }
            if (sym < 256) {
                b.drop(lc);
                return (unsigned)sym | 1u << 31;
            }
            base = sym == 256 ? 0 : len_base(sym - 257);
            x = sym == 256 ? 0 : len_extra(sym - 257);
        }
        b.drop(lc);
        if (base == 0) {
            in_block = 0;
            return 0u;
        }
        const unsigned len = (unsigned)base + (b.lo & ((1u << x) - 1u));
        b.drop(x);
        b.refill();
        const unsigned d = dist.fast[b.lo & kFastMask];
        int ld = (int)(d & 15u), xd = (int)((d >> 4) & 15u), db = (int)(d >> 8);
        if (ld == 0) {
            const int ds = long_code(dist, b.lo, ld);
            if (ds < 0 || ds > 29) {
                err = 17;
                return 0u;
            }
            xd = dist_extra(ds);
            db = dist_base(ds);
        }
        b.drop(ld);
        const unsigned m = len | ((unsigned)db + (b.lo & ((1u << xd) - 1u))) << 9;
        b.drop(xd);
        return m;
    }

    // Serial decoding: until `cap` matches are recorded (batch[i] =
    // {position, length, distance}), a
    // stored block's bytes are reached, the last block ends, or an error.
    // Literals go to dst directly; matches are for the caller to copy in
    // order, and so is a stored block (run_src, run_dst, run_n: input to
    // output, disjoint from the matches). Returns the number of matches
    // recorded. The GPU kernel has two warps share this work.
    CZ_MEM int step(uint8_t *dst, long long oend, int (*batch)[3], int cap, Huff &lit, Huff &dist,
                   unsigned char *lens)
    {
        int n = 0;
        run_n = 0;
        auto literal = [&](unsigned v) {
            if (op >= oend) err = 15;
            else dst[op++] = (uint8_t)v;
        };
        while (!err && n < cap) {
            if (!in_block) {
                if (final_block) break;
                if (block_header(lit.fast, lens)) break;
                if (btype != 0) {
                    if (!build(lit, lens, nlen, true)) err = 9;
                    else if (!build(dist, lens + nlen, ndist, false)) err = 10;
                    if (err) break;
                }
            }
            if (btype == 0) {
                if (op + stored_left > oend) {
                    err = 12;
                    break;
                }
                if (!stored_run()) break;
                run_dst = op;
                op += run_n;
                break;  // copied before the next step
            }
            const Record r = record(lit, dist);
            if (!err && b.over()) err = 14;
            for (int j = 0; j < 3 && !err; ++j)
                for (int i = 0; i < literals(r.e[j]) && !err; ++i) literal(r.e[j] >> (8 + 8 * i));
            if (err || r.m == 0) continue;
            if (r.m >> 31) {
                literal(r.m);
                continue;
            }
            const int len = (int)(r.m & 511u), d = (int)(r.m >> 9);
            if (d > op) {
                err = 19;
                break;
            }
            if (op + len > oend) {
                err = 20;
                break;
            }
            batch[n][0] = (int)op;
            batch[n][1] = len;
            batch[n][2] = d;
            ++n;
            op += len;
        }
        return n;
    }

    CZ_MEM bool done() const { return !in_block && final_block; }

    // After the last block: the big-endian Adler-32 (RFC 1950 2.2); err set
    // if it is missing.
    CZ_MEM unsigned trailer()
    {
        b.align();
        const unsigned t3 = b.get(8), t2 = b.get(8), t1 = b.get(8), t0 = b.get(8);
        if (b.over()) err = 21;
        return (t3 << 24) | (t2 << 16) | (t1 << 8) | t0;
    }
};

}  // namespace zl
}  // namespace cz
