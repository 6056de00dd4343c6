// cz_codec.cu -- the block codec kernels.
//
// encode: field blocks -> [int32 nbytes][4096-byte mask][survivors] records,
//   fusing the reference's WaveletCompressor::compress sequence
//   (WaveletCompressor.cpp:152-182): fwt (FullWaveletTransform.h:44-49),
//   threshold with the coarse-first survivor order (:58-96),
//   serialize_bitset (WaveletCompressor.cpp:96-122), float_zero_bits3
//   (:33-43) and shuffle3 (:55-73), plus the record framing of the writer's
//   block loop (SerializerIO_WaveletCompression_MPI_Simple.h:236-240).
// decode: records -> field blocks, the reference's decompress
//   (WaveletCompressor.cpp:231-259): deserialize_bitset, reshuffle3, load
//   (FullWaveletTransform.h:99-150) and iwt.
//
// One CTA of 512 threads per SM, persistent; blocks come from a device work
// queue, so one launch serves one field or a batch of uneven fields.
//
// What bounds these kernels is not memory (a block is 128 KB in, under 60 KB
// out) but one block's serial chain: nine sweeps, each needing the whole
// result of the one before, with the SM to itself (a block fills more than
// half of shared memory). So the chain is cut to five block-wide barriers:
//   * planes -- the x and y sweeps of level 32 only mix values of one z plane,
//     so a warp takes a plane through both on its own. Planes move between
//     the field and a ring of 4 KB slots by TMA (128-byte swizzle: the x
//     lines, one per lane, are read and written as 16-byte words without
//     bank conflicts); a consumed slot is refilled at once, which brings in
//     the next block while this one finishes.
//   * slabs -- the block lies as [y][z][x], so the z lines of one y are 4 KB
//     that belong to one warp. It transforms them, thresholds them (a lane's
//     line holds two runs of the survivor order) and packs the survivors of
//     each octant into a quarter of the same slab, so that they leave the SM
//     in stream order without a second pass over the block. The corner's z
//     lines continue through level 16 in registers, as the corner's y lines
//     later do through level 8.
//   * corner -- levels 16 and 8 (an eighth of the block) stay in the first
//     quarters of slabs 0..15 and are thresholded 8 positions per thread.
// The decoder runs the same steps backwards. Measured at 512^3 (wtype 1,
// threshold 1e-3 of the range): encode 0.664 -> 0.416 ms, decode 0.730 ->
// 0.431 ms against one thread-block-wide pass per sweep with row loads into
// registers (fourteen barriers a block, 16-byte loads and stores that touch
// 32 rows each).
#include "cz_block.cuh"
#include "cz_tma.cuh"

namespace cz {

// ------------------------------------------------------- shared memory map
constexpr int kMain = 0;                           // [y][z][x], 128 KB; slab y at 4096 y
constexpr int kPlane = 4096;                       // bytes of a z plane and of a slab
constexpr int kRing = kMain + 32 * kPlane;         // plane slots
constexpr int kSlots = 22;                         // what fits beside the block
constexpr int kStores = 16;                        // decode: one slot per warp
constexpr int kMaskAt = kRing + kSlots * kPlane;   // 4096 B, u32 words
constexpr int kSegCnt = kMaskAt + kMaskBytes;      // int x 112: survivors per (octant, slab) of level 32
constexpr int kWarpCnt = kSegCnt + 112 * 4;        // int x 16: survivors per warp of the corner
constexpr int kBlkAt = kWarpCnt + 64;              // Blk x 4
constexpr int kBarAt = kBlkAt + 4 * 32;            // mbarrier per slot
constexpr int kFailAt = kBarAt + 8 * kSlots;
constexpr int kBroughtAt = kFailAt + 16;           // encode: u32 per slot, 1 + the last plane brought into it
constexpr int kCodecSmem = kBroughtAt + 4 * kSlots;
constexpr int kMaskOdd = kRing + (kStores + 1) * kPlane;  // decode: the mask of every second block
constexpr int kRecAt = kRing + (kStores + 2) * kPlane;    // decode: Rec x 4
static_assert(kCodecSmem <= 232448, "shared memory of one CTA");
static_assert(kBarAt % 8 == 0 && kBlkAt % 8 == 0, "alignment");

// One block of the CTA's sequence; g < 0: no more.
struct Blk {
    long long g;
    int field, x, y, z;  // first sample
    float eps;
    int pad;
};
static_assert(sizeof(Blk) == 32, "Blk");

// Block g of the launch, and its field's tensor map made ready for the CTA: every
// use of it lies behind a CTA-wide barrier after this.
__device__ __forceinline__ void set_block(Blk *b, long long g, const CzFields &fs, long long total)
{
    b->g = -1;
    if (g < total) {
        const CzField *fields = fs.list ? fs.list : &fs.one;
        const BlockRef r = locate(fields, fs.n, g);
        b->field = (int)(r.f - fields);
        if (fs.list) tma_map_acquire(fs.maps + b->field);
        b->x = 32 * r.bx;
        b->y = 32 * r.by;
        b->z = 32 * r.bz;
        b->eps = r.f->eps;
        b->g = g;
    }
}

// The CTA's blocks come from the queue, the second one with the first; where
// every block can have a CTA of its own, without it.
__device__ __forceinline__ void take_first(Blk *b, const CzFields &fs, long long total, unsigned long long *queue)
{
    const long long g = total <= gridDim.x ? (long long)blockIdx.x : (long long)atomicAdd(queue, 1ull);
    set_block(b, g, fs, total);
}
__device__ __forceinline__ void take_later(Blk *b, const CzFields &fs, long long total, unsigned long long *queue)
{
    if (total > gridDim.x) set_block(b, (long long)atomicAdd(queue, 1ull), fs, total);
    else b->g = -1;
}

// Named barrier of the first n threads (whole warps).
template <int ID, int N>
__device__ __forceinline__ void bar_first()
{
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}

// Survivor q of a 1 KB quarter (byte address p = base + 4 q) sits at
// quarter(p): 16 lanes that write 16 consecutive survivors each (a dense
// region) then hit 16 different banks, and 32 lanes that read consecutive
// survivors 32.
__device__ __forceinline__ uint32_t quarter(uint32_t p) { return p ^ ((p >> 4) & 0x3cu); }

// Corner coefficient (x, y, z), all < 16, of the block.
__device__ __forceinline__ int corner(int x, int y, int z) { return kMain + y * kPlane + z * 64 + ((x ^ z) & 15) * 4; }

__device__ __forceinline__ float &at(unsigned char *sm, uint32_t byte) { return *reinterpret_cast<float *>(sm + byte); }

// x line of a plane slot (row = lane), 16-byte words behind the TMA's
// 128-byte swizzle (word c of row r at c ^ (r & 7)).
__device__ __forceinline__ void ld_row(const unsigned char *slot, int row, float (&v)[32])
{
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float4 q = *reinterpret_cast<const float4 *>(slot + row * 128 + ((c ^ (row & 7)) << 4));
        v[4 * c] = q.x;
        v[4 * c + 1] = q.y;
        v[4 * c + 2] = q.z;
        v[4 * c + 3] = q.w;
    }
}
__device__ __forceinline__ void st_row(unsigned char *slot, int row, const float (&v)[32])
{
#pragma unroll
    for (int c = 0; c < 8; ++c)
        *reinterpret_cast<float4 *>(slot + row * 128 + ((c ^ (row & 7)) << 4)) =
            make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}
// y line of a plane slot (column x).
__device__ __forceinline__ uint32_t col_at(int x, int y)
{
    return (uint32_t)(y * 128 + (((x >> 2) ^ (y & 7)) << 4) + (x & 3) * 4);
}

// The 8 positions of the corner that thread t holds in stream order (stream
// indices 8t .. 8t+7, FullWaveletTransform.h:63-93): the coarse 4^3 (t < 8),
// two runs of 4 along x of level 8 (t < 64), one run of 8 along y of level
// 16. f(e, x, y, z) for e = 0..7.
template <class F>
__device__ __forceinline__ void corner_run(int t, F &&f)
{
    if (t < 8) {
#pragma unroll
        for (int e = 0; e < 8; ++e) f(e, e & 3, 2 * (t & 1) + (e >> 2), t >> 1);
    } else if (t < 64) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int q = 2 * (t - 8) + (e >> 2), c = (q >> 4) + 1;
            f(e, 4 * (c & 1) + (e & 3), 4 * ((c >> 1) & 1) + (q & 3), 4 * (c >> 2) + ((q >> 2) & 3));
        }
    } else {
        const int q = t - 64, c = (q >> 6) + 1;
#pragma unroll
        for (int e = 0; e < 8; ++e) f(e, 8 * (c >> 2) + ((q >> 3) & 7), 8 * (c & 1) + e, 8 * ((c >> 1) & 1) + (q & 7));
    }
}

// Inclusive sums within each half warp.
__device__ __forceinline__ int half_scan(int c, int lane)
{
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, c, o, 16);
        if ((lane & 15) >= o) c += t;
    }
    return c;
}
__device__ __forceinline__ int warp_scan(int c, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) c += t;
    }
    return c;
}

// Stream offsets once every count is in shared memory: where the warp's
// part of the corner starts, the corner's total, and the survivors before
// each of the 112 level-32 segments (order: octant code, then y).
struct Offsets {
    int mine, corner, total, seg;  // seg: exclusive sum of segment 4 lane + (warp & 3)
    __device__ __forceinline__ int of(int code, int warp) const
    {
        return corner + __shfl_sync(0xffffffffu, seg, (code - 1) * 4 + (warp >> 2));
    }
};
__device__ __forceinline__ Offsets stream_offsets(const unsigned char *sm, int warp, int lane)
{
    const int *wc = reinterpret_cast<const int *>(sm + kWarpCnt);
    const int n = lane < kNW ? wc[lane] : 0, in = warp_scan(n, lane);
    Offsets o;
    o.mine = __shfl_sync(0xffffffffu, in - n, warp);
    o.corner = __shfl_sync(0xffffffffu, in, 31);
    int4 c = make_int4(0, 0, 0, 0);
    if (lane < 28) c = reinterpret_cast<const int4 *>(sm + kSegCnt)[lane];
    const int s = c.x + c.y + c.z + c.w, si = warp_scan(s, lane), k = warp & 3;
    o.total = o.corner + __shfl_sync(0xffffffffu, si, 31);
    o.seg = si - s + (k > 0 ? c.x : 0) + (k > 1 ? c.y : 0) + (k > 2 ? c.z : 0);
    return o;
}

// ------------------------------------------------------------------ encode
// Bit j: |v[j]| > eps (FullWaveletTransform.h:84), eps not -0, as the sign of
// eps - |v[j]| (rounding keeps a difference's sign; a NaN's is clear): one
// ALU instruction per value, where a compare and an OR take two.
template <int N>
__device__ __forceinline__ unsigned keep_line(const float (&v)[N], float eps)
{
    unsigned b = 0;
#pragma unroll
    for (int j = N - 1; j >= 0; --j) b = __funnelshift_l(__float_as_uint(__fadd_rn(eps, -fabsf(v[j]))), b, 1);
    return b;
}

// Survivors j of a lane's line whose keep bit is set, in order, to the
// quarter at shared address p. Predicated: as branches the 64 tests of a
// line took 15 instructions each.
template <int J0>
__device__ __forceinline__ void pack16(uint32_t p, unsigned bits, const float (&v)[32])
{
#pragma unroll
    for (int j = 0; j < 16; ++j)
        asm volatile("{\n .reg .pred q;\n .reg .b32 t;\n setp.ne.u32 q, %1, 0;\n"
                     " shr.u32 t, %0, 4;\n and.b32 t, t, 60;\n xor.b32 t, t, %0;\n"
                     " @q st.shared.f32 [t], %2;\n @q add.u32 %0, %0, 4;\n}"
                     : "+r"(p)
                     : "r"(bits & (1u << j)), "f"(v[J0 + j])
                     : "memory");
}

// n survivors of the quarter at p to stream positions k0 ..: zero bits, byte
// planes S apart when shuffling.
__device__ __forceinline__ void emit_quarter(unsigned char *sm, uint32_t p, int n, uint8_t *pay, int k0, int S,
                                             uint32_t zmask, int shuffle, int lane)
{
    if (shuffle) {
        uint8_t *d0 = pay + k0, *d1 = d0 + S, *d2 = d1 + S, *d3 = d2 + S;
        for (int b = lane; b < n; b += 32) {
            const uint32_t u = __float_as_uint(at(sm, quarter(p + 4 * b))) & zmask;
            d0[b] = (uint8_t)u;
            d1[b] = (uint8_t)(u >> 8);
            d2[b] = (uint8_t)(u >> 16);
            d3[b] = (uint8_t)(u >> 24);
        }
    } else {
        uint32_t *d = reinterpret_cast<uint32_t *>(pay) + k0;
        for (int b = lane; b < n; b += 32) d[b] = __float_as_uint(at(sm, quarter(p + 4 * b))) & zmask;
    }
}

// AHEAD: the planes of the next block that do not fit the ring are brought
// into L2 while this block is finished (the autotuner times both).
template <int KIND, bool AHEAD>
__global__ void __launch_bounds__(kNT, 1)
encode_kernel(const __grid_constant__ CzFields fs, long long total_blocks, int zerobits, int shuffle, uint8_t *stage,
              int *rec_bytes, unsigned long long *queue, int *err, CzChunks chunks)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t zmask = zerobits > 0 ? ~((1u << zerobits) - 1u) : 0xffffffffu;
    uint32_t *mask32 = reinterpret_cast<uint32_t *>(sm + kMaskAt);
    int *seg_cnt = reinterpret_cast<int *>(sm + kSegCnt), *warp_cnt = reinterpret_cast<int *>(sm + kWarpCnt);
    Blk *blk = reinterpret_cast<Blk *>(sm + kBlkAt);
    volatile int *fail = reinterpret_cast<volatile int *>(sm + kFailAt);
    uint32_t *brought = reinterpret_cast<uint32_t *>(sm + kBroughtAt);
    const uint32_t bars = smem_u32(sm + kBarAt), ring = smem_u32(sm + kRing);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(bars + 8 * s, 1);
            brought[s] = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *fail = 0;
        take_first(blk, fs, total_blocks, queue);
    }
    __syncthreads();
    // plane n of the CTA's sequence (plane n & 31 of its block n >> 5) into
    // its slot, by one lane
    auto bring = [&](uint32_t n) {
        const Blk &b = blk[(n >> 5) & 3];
        if (b.g < 0) return;
        const uint32_t s = n % kSlots;
        brought[s] = n + 1;
        tma_load_3d(ring + s * kPlane, fs.list ? fs.maps + b.field : &fs.map, b.x, b.y, b.z + (int)(n & 31), bars + 8 * s,
                    kPlane);
    };
    if (lane == 0) {
        bring(warp);
        if (warp + 16 < kSlots) bring(warp + 16);
    }
    if (threadIdx.x == 0) take_later(blk + 1, fs, total_blocks, queue);
    __syncthreads();

    uint32_t it = 0;
    for (;; ++it) {
        const Blk &cur = blk[it & 3];
        const long long g = cur.g;
        if (g < 0) break;
        const float eps = cur.eps + 0.f;  // a threshold of -0 as 0
        // ---- level 32, x then y: planes z = warp and warp + 16
#pragma unroll 1
        for (int r = 0; r < 2; ++r) {
            const int z = warp + 16 * r;
            const uint32_t n = 32 * it + z, s = n % kSlots;
            unsigned char *slot = sm + kRing + s * kPlane;
            // after one wait ran out the others poll only briefly: the CTA
            // ends, and its error is reported
            const bool here = mbar_wait(bars + 8 * s, (n / kSlots) & 1, *fail ? 64 : kTilePolls);
            if (!here) *fail = 1;
            float v[32];
            ld_row(slot, lane, v);
            line_fwd<32, KIND>(v);
            st_row(slot, lane, v);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = at(slot, col_at(lane, j));
            __syncwarp();
            // a slot whose copy is still to come gets no second one: planes 22 to 31
            // follow planes 0 to 9 of the same block, whose waits are over at r == 1
            if (lane == 0 && here && !*fail) {
                fence_async_smem();
                bring(n + kSlots);
            }
            line_fwd<32, KIND>(v);
            if (r == 0) __syncthreads();  // the previous block has left the slabs
#pragma unroll
            for (int j = 0; j < 32; ++j) at(sm, kMain + j * kPlane + z * 128 + lane * 4) = v[j];
        }
        __syncthreads();
        if (*fail) break;  // the same for all: the waits are over until the next block
        // ---- level 32, z: slabs y = warp and warp + 16
#pragma unroll 1
        for (int r = 0; r < 2; ++r) {
            const int y = warp + 16 * r;
            const uint32_t slab = kMain + y * kPlane;
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = at(sm, slab + j * 128 + lane * 4);
            __syncwarp();
            line_fwd<32, KIND>(v);
            const bool in_corner = r == 0 && lane < 16;
            unsigned kb = keep_line(v, eps);
            if (in_corner) kb &= 0xffff0000u;
            mask32[lane + 32 * y] = kb;  // positional word y*32+x, bits z
            // quarters: code & 3 = (z >= 16) | (x >= 16) << 1
            const int c = __popc(kb & 0xffffu) | __popc(kb >> 16) << 16;
            const int in = half_scan(c, lane), ex = in - c;
            const int xh = lane >> 4, code = (xh << 1) | (r << 2);
            if ((lane & 15) == 15) {
                if (code) seg_cnt[(code - 1) * 16 + warp] = in & 0xffff;
                seg_cnt[code * 16 + warp] = in >> 16;
            }
            const uint32_t q = smem_u32(sm) + slab + xh * 2048;
            pack16<0>(q + (ex & 0xffff) * 4, kb & 0xffffu, v);
            pack16<16>(q + 1024 + (ex >> 16) * 4, kb >> 16, v);
            if (r == 0) {  // the corner's z lines go on through level 16
                float u[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) u[j] = v[j];
                line_fwd<16, KIND>(u);
                if (lane < 16) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) at(sm, corner(lane, y, j)) = u[j];
                }
            }
        }
        __syncthreads();
        if (warp == kNW - 1 && lane == 0) take_later(blk + ((it + 2) & 3), fs, total_blocks, queue);
        if (AHEAD && warp == kNW - 2 && lane >= kSlots) {
            const Blk &b = blk[(it + 1) & 3];
            if (b.g >= 0) tma_prefetch_3d(fs.list ? fs.maps + b.field : &fs.map, b.x, b.y, b.z + lane);
        }
        if (warp < 8) {
            // ---- level 16, x (lines (y, z)) and y (lines (x, z)), level 8, y
            float u[16];
            {
                const int z = lane & 15, y = 2 * warp + (lane >> 4);
#pragma unroll
                for (int j = 0; j < 16; ++j) u[j] = at(sm, corner(j, y, z));
                line_fwd<16, KIND>(u);
#pragma unroll
                for (int j = 0; j < 16; ++j) at(sm, corner(j, y, z)) = u[j];
            }
            bar_first<1, 256>();
            {
                const int z = lane & 15, x = 2 * warp + (lane >> 4);
#pragma unroll
                for (int j = 0; j < 16; ++j) u[j] = at(sm, corner(x, j, z));
                line_fwd<16, KIND>(u);
                const unsigned kb = keep_line(u, eps);
                // positional word x*32+z, bits y; the 8^3 corner's low byte comes later
                if (x < 8 && z < 8) reinterpret_cast<uint8_t *>(mask32)[4 * (z + 32 * x) + 1] = (uint8_t)(kb >> 8);
                else reinterpret_cast<uint16_t *>(mask32)[2 * (z + 32 * x)] = (uint16_t)kb;
                if (warp < 4) {
                    float w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) w[j] = u[j];
                    line_fwd<8, KIND>(w);
                    if (z < 8) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) u[j] = w[j];
                    }
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) at(sm, corner(x, j, z)) = u[j];
            }
            if (warp < 4) bar_first<2, 128>();
            if (warp < 2) {
                // ---- level 8, z then x
                float w[8];
                {
                    const int x = lane & 7, y = 4 * warp + (lane >> 3);
#pragma unroll
                    for (int j = 0; j < 8; ++j) w[j] = at(sm, corner(x, y, j));
                    line_fwd<8, KIND>(w);
#pragma unroll
                    for (int j = 0; j < 8; ++j) at(sm, corner(x, y, j)) = w[j];
                }
                bar_first<3, 64>();
                const int y = lane & 7, z = 4 * warp + (lane >> 3);
#pragma unroll
                for (int j = 0; j < 8; ++j) w[j] = at(sm, corner(j, y, z));
                line_fwd<8, KIND>(w);
#pragma unroll
                for (int j = 0; j < 8; ++j) at(sm, corner(j, y, z)) = w[j];
                unsigned kb = keep_line(w, eps);
                if (y < 4 && z < 4) kb |= 0xFu;  // the coarse 4^3 is always kept (FullWaveletTransform.h:165-168)
                reinterpret_cast<uint8_t *>(mask32)[4 * (y + 32 * z)] = (uint8_t)kb;
            }
        }
        __syncthreads();
        // ---- the corner's survivors, 8 stream positions per thread
        float u[8];
        corner_run((int)threadIdx.x, [&](int e, int x, int y, int z) { u[e] = at(sm, corner(x, y, z)); });
        unsigned kc = keep_line(u, eps);
        if (threadIdx.x < 8) kc = 0xffu;
        const int nc = __popc(kc), inc = warp_scan(nc, lane);
        if (lane == 31) warp_cnt[warp] = inc;
        __syncthreads();
        const Offsets of = stream_offsets(sm, warp, lane);
        const int S = of.total, nb = kMaskBytes + 4 * S;
        uint8_t *rec = stage + (size_t)g * kSlotBytes, *pay = rec + 4 + kMaskBytes;
        if (threadIdx.x == 0) {
            *reinterpret_cast<int *>(rec) = nb;
            rec_bytes[g] = nb;
            record_done(chunks, g, nb);
        }
        for (int i = threadIdx.x; i < kMaskBytes / 4; i += kNT) reinterpret_cast<uint32_t *>(rec + 4)[i] = mask32[i];
        {
            // the corner has been read: its first quarters take its survivors
            const uint32_t q = kMain + warp * kPlane;
            uint32_t p = q + 4 * (inc - nc);
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (kc & (1u << e)) {
                    at(sm, quarter(p)) = u[e];
                    p += 4;
                }
            const int n = __shfl_sync(0xffffffffu, inc, 31);
            __syncwarp();
            emit_quarter(sm, q, n, pay, of.mine, S, zmask, shuffle, lane);
        }
#pragma unroll 1
        for (int code = 1; code < 8; ++code) {
            const int y = warp + 16 * (code >> 2), n = seg_cnt[(code - 1) * 16 + warp];
            emit_quarter(sm, kMain + y * kPlane + (code & 3) * 1024, n, pay, of.of(code, warp), S, zmask, shuffle,
                         lane);
        }
    }
    // every plane brought in was waited for; a CTA that gave up waiting lets its
    // copies land (bounded) before it leaves, and gives the blocks that it has
    // taken, and those that nobody has yet, the sizes that what follows reads
    if (*fail && threadIdx.x == 0) {
        if (err) atomicExch(err, 1);
        for (uint32_t s = 0; s < kSlots; ++s)
            if (brought[s]) mbar_wait(bars + 8 * s, ((brought[s] - 1) / kSlots) & 1);
        auto skip = [&](long long g) {
            *reinterpret_cast<int *>(stage + (size_t)g * kSlotBytes) = kMaskBytes;
            rec_bytes[g] = kMaskBytes;
            record_done(chunks, g, kMaskBytes);
        };
        for (uint32_t k = it; k < it + 2; ++k)
            if (blk[k & 3].g >= 0) skip(blk[k & 3].g);
        if (total_blocks > gridDim.x)
            for (long long g; (g = (long long)atomicAdd(queue, 1ull)) < total_blocks;) skip(g);
    }
}

// Error statistics of a decoded block against a reference field (the
// quantities of cz2diff, Tools/cz2diff.cpp:116-261): per block
// {e_inf, n_inf, e_1, n_1, e_2, n_2, min, max} with e = |decoded - ref|,
// n = |ref|. The difference is exact (two-sum), maxima are exact, the sums
// are compensated binary32 per thread and binary64 beyond.
struct DiffAcc {
    float es = 0.f, ee = 0.f;  // largest error as s + e (two-sum parts)
    float ninf = 0.f, mn = 3.4e38f, mx = -3.4e38f;
    float s[4] = {0.f, 0.f, 0.f, 0.f}, c[4] = {0.f, 0.f, 0.f, 0.f};  // e_1, e_2, n_1, n_2 (Neumaier)
    __device__ __forceinline__ void add(int k, float x)
    {
        const float t = __fadd_rn(s[k], x);
        c[k] = __fadd_rn(c[k], fabsf(s[k]) >= fabsf(x) ? __fadd_rn(__fsub_rn(s[k], t), x)
                                                       : __fadd_rn(__fsub_rn(x, t), s[k]));
        s[k] = t;
    }
    __device__ __forceinline__ void put(float f1, float f2)
    {
        // TwoSum(f1, -f2): d + r == f1 - f2 exactly
        const float d = __fadd_rn(f1, -f2);
        const float bv = __fsub_rn(d, f1);
        const float av = __fsub_rn(d, bv);
        const float r = __fadd_rn(__fsub_rn(f1, av), __fsub_rn(-f2, bv));
        const float a = fabsf(d);
        if (a > fabsf(es) || (a == fabsf(es) && fabs((double)d + r) > fabs((double)es + ee))) {
            es = d;
            ee = r;
        }
        const float n = fabsf(f2);
        ninf = fmaxf(ninf, n);
        mn = fminf(mn, f2);
        mx = fmaxf(mx, f2);
        // every term with its rounding error: |e| = a + sgn(d) r,
        // e^2 = a*a (+ fma residual) + 2 a sgn(d) r, n^2 = n*n (+ residual)
        const float sr = d >= 0.f ? r : -r;
        add(0, a);
        add(0, sr);
        const float a2 = __fmul_rn(a, a);
        add(1, a2);
        add(1, __fmaf_rn(a, a, -a2));
        add(1, __fmul_rn(2.f * a, sr));
        add(2, n);
        const float n2 = __fmul_rn(n, n);
        add(3, n2);
        add(3, __fmaf_rn(n, n, -n2));
    }
};

// ------------------------------------------------------------------ decode
// Where a block's record is.
struct Rec {
    const uint8_t *rec, *q12;  // record; byte planes 1 and 2 left in the LZ4 input (or null)
    int nb, ok;                // record bytes; whether they can be a record's
};

// Four bytes of each plane of a shuffled payload, as read: survivors k + j ..
// k + j + 3 (j < n wanted, j a multiple of 4) from two aligned words per
// plane; every load is of a word that holds a wanted byte. The words' place
// within the aligned ones depends on k and the plane alone.
struct Raw {
    uint32_t lo[4], hi[4];
};
__device__ __forceinline__ const uint8_t *plane_at(const Payload &pl, int i, int k)
{
    return (i == 0 ? pl.p : i == 1 ? pl.q : i == 2 ? pl.q + pl.c : pl.p + 3 * pl.c) + k;
}
__device__ __forceinline__ void planes_load(const Payload &pl, int k, int j, int n, Raw &r)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(plane_at(pl, i, k));
        const int off = (int)(a & 3);
        const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3) + ((unsigned)j >> 2);
        r.lo[i] = j < n ? __ldg(w) : 0u;
        r.hi[i] = off && j + 4 - off < n ? __ldg(w + 1) : 0u;
    }
}
// ... and into the quarter whose first survivor is k's, at p.
__device__ __forceinline__ void planes_store(unsigned char *sm, uint32_t p, const Payload &pl, int k, int j, int n,
                                             const Raw &r)
{
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = __funnelshift_r(r.lo[i], r.hi[i], 8 * (uint32_t)(reinterpret_cast<uintptr_t>(plane_at(pl, i, k)) & 3));
    const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[0], w[1], 0x7362);
    const uint32_t c = __byte_perm(w[2], w[3], 0x5140), d = __byte_perm(w[2], w[3], 0x7362);
    const uint32_t at0 = quarter(p + 4 * j);  // the four share the swizzle
    if (j < n) at(sm, at0) = __uint_as_float(__byte_perm(a, c, 0x5410));
    if (j + 1 < n) at(sm, at0 ^ 4) = __uint_as_float(__byte_perm(a, c, 0x7632));
    if (j + 2 < n) at(sm, at0 ^ 8) = __uint_as_float(__byte_perm(b, d, 0x5410));
    if (j + 3 < n) at(sm, at0 ^ 12) = __uint_as_float(__byte_perm(b, d, 0x7632));
}

// A lane's run from its quarter at shared address p: survivor or zero at
// each place.
template <int J0>
__device__ __forceinline__ void unpack16(uint32_t p, unsigned bits, float (&v)[32])
{
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float x = 0.f;
        asm volatile("{\n .reg .pred q;\n .reg .b32 t;\n setp.ne.u32 q, %2, 0;\n"
                     " shr.u32 t, %0, 4;\n and.b32 t, t, 60;\n xor.b32 t, t, %0;\n"
                     " @q ld.shared.f32 %1, [t];\n @q add.u32 %0, %0, 4;\n}"
                     : "+r"(p), "+f"(x)
                     : "r"(bits & (1u << j))
                     : "memory");
        v[J0 + j] = x;
    }
}

__device__ __forceinline__ double diff_fold(int k, double r, double x)
{
    return (k == 0 || k == 1 || k == 7) ? fmax(r, x) : (k == 6 ? fmin(r, x) : r + x);
}
// Four quantities over the warp by f, quantity k in lane 8 k. Halves of the warp
// take two each, quarters one (6 operations instead of 20; binary64 runs at 2
// lanes a cycle and SM), in the order of a butterfly over all lanes.
template <class F>
__device__ __forceinline__ double warp_fold4(double a0, double a1, double a2, double a3, F &&f)
{
    const int lane = threadIdx.x & 31;
    const bool h = lane & 16, q = lane & 8;
    const double b0 = f(h ? a2 : a0, __shfl_xor_sync(0xffffffffu, h ? a0 : a2, 16));
    const double b1 = f(h ? a3 : a1, __shfl_xor_sync(0xffffffffu, h ? a1 : a3, 16));
    double c = f(q ? b1 : b0, __shfl_xor_sync(0xffffffffu, q ? b0 : b1, 8));
#pragma unroll
    for (int o = 4; o; o >>= 1) c = f(c, __shfl_xor_sync(0xffffffffu, c, o));
    return c;
}

template <int KIND, bool DIFF>
__global__ void __launch_bounds__(kNT, 1)
decode_kernel(const __grid_constant__ CzFields fs, long long total_blocks, int shuffle, CzRecords where, int *flag,
              unsigned long long *queue, const float *diff_ref, double *diff_out, CzPlanes planes)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int *seg_cnt = reinterpret_cast<int *>(sm + kSegCnt), *warp_cnt = reinterpret_cast<int *>(sm + kWarpCnt);
    Blk *blk = reinterpret_cast<Blk *>(sm + kBlkAt);
    Rec *recs = reinterpret_cast<Rec *>(sm + kRecAt);
    volatile int *bad = reinterpret_cast<volatile int *>(sm + kFailAt);  // per parity of the block's number
    unsigned char *slot = sm + kRing + warp * kPlane;  // this warp's plane
    // Record of block n of the CTA's sequence in two steps, so that none of
    // the dependent loads (offset, byte count, mask) waits on its own: where
    // it is ...
    auto find = [&](uint32_t n, long long ro, long long len, int nb, const int4 &hole, long long src_off) {
        const uint8_t *rec = where.base + (ro < 0 ? 0 : ro), *q12 = nullptr;
        const bool ok = nb >= kMaskBytes && nb <= kMaxRecord + 4 && 4 + nb <= len;
        // byte planes 1 and 2 where the LZ4 stage left them in its input
        const int c4 = (nb - kMaskBytes) / 4;
        if (ok && hole.z > 0 && hole.z == 2 * c4 && hole.x == 4 + kMaskBytes + c4) q12 = planes.src + src_off + hole.y;
        recs[n & 3] = Rec{rec, q12, nb, ok};
    };
    const bool holes = planes.hole != nullptr && shuffle;
    // ... then, by threads t of nt, its mask (deserialize_bitset,
    // WaveletCompressor.cpp:124-150) into shared memory, its payload into L2.
    auto fetch = [&](uint32_t n, int t, int nt) {
        const Rec r = recs[n & 3];
        uint32_t *m = reinterpret_cast<uint32_t *>(sm + (n & 1 ? kMaskOdd : kMaskAt));
#pragma unroll 5
        for (int i = t; i < kMaskBytes / 4; i += nt)
            m[i] = r.ok ? __ldg(reinterpret_cast<const uint32_t *>(r.rec + 4) + i) : 0u;
        if (r.ok) prefetch_record(r.rec, r.nb, r.q12, t, nt);
    };
    // the block after next, by the last warp's first lane: its ticket, record
    // offset, byte count and planes, each loaded in one phase of the block
    // and used in a later one
    const bool scout = threadIdx.x == 32 * (kNW - 1);
    unsigned long long s_ticket = 0;
    long long s_off = -1, s_len = 0, s_src = 0;  // s_len: bytes from there on that can be the record's
    int s_nb = -1;
    int4 s_hole = make_int4(0, 0, 0, 0);
    auto scout_off = [&](uint32_t n) {
        const long long g = blk[n & 3].g;
        s_off = -1;
        s_len = 0x7fffffff;
        if (g < 0) return;
        if (where.rec_off) {
            s_off = where.rec_off[g];
        } else if (where.cap) {
            s_off = g * where.cap;
            s_len = where.dec_len[g];
        } else {
            s_off = where.off[g];
            s_len = where.off[g + 1] - s_off;
        }
        if (s_len < 4 || s_len > 0x7fffffff) s_off = -1;
    };
    auto scout_rec = [&](uint32_t n) {
        const long long g = blk[n & 3].g;
        s_nb = s_off >= 0 ? *reinterpret_cast<const int *>(where.base + s_off) : -1;
        if (g >= 0 && holes) {
            s_hole = planes.hole[g];
            s_src = planes.src_off[g];
        }
    };
    if (scout) {
        bad[0] = bad[1] = 0;
        take_first(blk, fs, total_blocks, queue);
        scout_off(0);
        scout_rec(0);
        find(0, s_off, s_len, s_nb, s_hole, s_src);
    }
    __syncthreads();
    if (blk[0].g < 0) return;
    if (scout) {
        take_later(blk + 1, fs, total_blocks, queue);
        scout_off(1);
        scout_rec(1);
        find(1, s_off, s_len, s_nb, s_hole, s_src);
    } else if (warp < kNW - 1) {
        fetch(0, threadIdx.x, kNT - 32);
    }
    __syncthreads();
    for (uint32_t it = 0;; ++it) {
        const Blk &cur = blk[it & 3];
        const long long g = cur.g;
        if (g < 0) break;
        const uint32_t *mask32 = reinterpret_cast<const uint32_t *>(sm + (it & 1 ? kMaskOdd : kMaskAt));
        const uint8_t *rec = recs[it & 3].rec, *q12 = recs[it & 3].q12;
        const int nb = recs[it & 3].nb;
        const bool more = blk[(it + 1) & 3].g >= 0;
        if (scout && more) s_ticket = atomicAdd(queue, 1ull);
        const bool size_ok = recs[it & 3].ok != 0;
        // ---- survivor counts: level 32 per (octant, slab), the corner per warp
        unsigned kz[2];
        int ex[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            kz[r] = mask32[lane + 32 * (warp + 16 * r)];
            if (r == 0 && lane < 16) kz[r] &= 0xffff0000u;
            const int c = __popc(kz[r] & 0xffffu) | __popc(kz[r] >> 16) << 16;
            const int in = half_scan(c, lane);
            ex[r] = in - c;
            const int code = ((lane >> 4) << 1) | (r << 2);
            if ((lane & 15) == 15) {
                if (code) seg_cnt[(code - 1) * 16 + warp] = in & 0xffff;
                seg_cnt[code * 16 + warp] = in >> 16;
            }
        }
        unsigned kc = 0;
        corner_run((int)threadIdx.x, [&](int e, int x, int y, int z) {
            const int b = threadIdx.x < 64 ? 32 * (y + 32 * z) + x : 32 * (z + 32 * x) + y;
            kc |= ((mask32[b >> 5] >> (b & 31)) & 1u) << e;
        });
        // the base case consumes exactly the 64 coarse survivors (:178-189)
        if (threadIdx.x < 8 && kc != 0xffu) bad[it & 1] = 1;
        const int nc = __popc(kc), inc = warp_scan(nc, lane);
        if (lane == 31) warp_cnt[warp] = inc;
        __syncthreads();
        const Offsets of = stream_offsets(sm, warp, lane);
        const int expected = of.total, payload = nb - kMaskBytes;
        int nel = payload / 4;
        if (nel - expected == 1) nel--;  // :247-250
        const bool ok = size_ok && nel == expected && !bad[it & 1];
        if (threadIdx.x == 0) {
            if (!ok) atomicMin(flag, -1);
            bad[(it + 1) & 1] = 0;
        }
        // ---- load (FullWaveletTransform.h:99-150): the survivors of every
        // quarter in stream order; a bad record decodes as an empty one
        if (ok) {
            Payload pl;
            pl.p = rec + 4 + kMaskBytes;
            pl.c = payload / 4;
            pl.q = q12 ? q12 : pl.p + pl.c;  // planes 1 and 2
            pl.shuffle = shuffle != 0;
            if (lane == 0) tma_store_wait_read();  // the slot holds the warp's corner survivors next
            __syncwarp();
            // list 0: the warp's part of the corner; 1-7: an octant's quarter
            auto list = [&](int code, uint32_t &p, int &n, int &k0) {
                p = code ? kMain + (warp + 16 * (code >> 2)) * kPlane + (code & 3) * 1024 : kRing + warp * kPlane;
                n = code ? seg_cnt[(code - 1) * 16 + warp] : warp_cnt[warp];
                const int seg = of.of(code ? code : 1, warp);
                k0 = code ? seg : of.mine;
            };
            uint32_t p;
            int n, k0;
            list(0, p, n, k0);
            if (pl.shuffle) {
                // 128 survivors a step, the next list's first step in flight
                // while this one's are placed
                Raw now;
                planes_load(pl, k0, 4 * lane, n, now);
#pragma unroll 1
                for (int code = 0; code < 8; ++code) {
                    uint32_t pn = 0;
                    int nn = 0, kn = 0;
                    if (code < 7) list(code + 1, pn, nn, kn);
                    Raw ahead;
                    planes_load(pl, kn, 4 * lane, nn, ahead);
                    if (n > 128) {
                        Raw more4;
                        planes_load(pl, k0, 128 + 4 * lane, n, more4);
                        planes_store(sm, p, pl, k0, 4 * lane, n, now);
                        planes_store(sm, p, pl, k0, 128 + 4 * lane, n, more4);
                    } else {
                        planes_store(sm, p, pl, k0, 4 * lane, n, now);
                    }
                    now = ahead;
                    p = pn;
                    n = nn;
                    k0 = kn;
                }
            } else {
                const float *src = reinterpret_cast<const float *>(pl.p);
#pragma unroll 1
                for (int code = 0; code < 8; ++code) {
                    if (code) list(code, p, n, k0);
#pragma unroll 4
                    for (int b = lane; b < n; b += 32) at(sm, quarter(p + 4 * b)) = __ldg(src + k0 + b);
                }
            }
        } else {
            kc = kz[0] = kz[1] = 0;
        }
        __syncwarp();
        {
            uint32_t p = kRing + warp * kPlane + 4 * (inc - nc);
            corner_run((int)threadIdx.x, [&](int e, int x, int y, int z) {
                float c = 0.f;
                if (kc & (1u << e)) {
                    c = at(sm, quarter(p));
                    p += 4;
                }
                at(sm, corner(x, y, z)) = c;
            });
        }
        __syncthreads();
        if (warp < 8) {
            // ---- level 8: x, z, then y with level 16's y and x
            float u[16];
            if (warp < 2) {
                float w[8];
                {
                    const int y = lane & 7, z = 4 * warp + (lane >> 3);
#pragma unroll
                    for (int j = 0; j < 8; ++j) w[j] = at(sm, corner(j, y, z));
                    line_inv<8, KIND>(w);
#pragma unroll
                    for (int j = 0; j < 8; ++j) at(sm, corner(j, y, z)) = w[j];
                }
                bar_first<3, 64>();
                const int x = lane & 7, y = 4 * warp + (lane >> 3);
#pragma unroll
                for (int j = 0; j < 8; ++j) w[j] = at(sm, corner(x, y, j));
                line_inv<8, KIND>(w);
#pragma unroll
                for (int j = 0; j < 8; ++j) at(sm, corner(x, y, j)) = w[j];
            }
            if (warp < 4) bar_first<2, 128>();
            {
                const int z = lane & 15, x = 2 * warp + (lane >> 4);
#pragma unroll
                for (int j = 0; j < 16; ++j) u[j] = at(sm, corner(x, j, z));
                if (warp < 4) {
                    float w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) w[j] = u[j];
                    line_inv<8, KIND>(w);
                    if (z < 8) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) u[j] = w[j];
                    }
                }
                line_inv<16, KIND>(u);
#pragma unroll
                for (int j = 0; j < 16; ++j) at(sm, corner(x, j, z)) = u[j];
            }
            bar_first<1, 256>();
            const int z = lane & 15, y = 2 * warp + (lane >> 4);
#pragma unroll
            for (int j = 0; j < 16; ++j) u[j] = at(sm, corner(j, y, z));
            line_inv<16, KIND>(u);
#pragma unroll
            for (int j = 0; j < 16; ++j) at(sm, corner(j, y, z)) = u[j];
        } else if (scout) {  // idle meanwhile
            blk[(it + 2) & 3].g = -1;
            if (more) set_block(blk + ((it + 2) & 3), (long long)s_ticket, fs, total_blocks);
            scout_off(it + 2);
        } else if (more && warp < kNW - 1) {
            fetch(it + 1, threadIdx.x - 256, kNT - 256 - 32);
        }
        __syncthreads();
        if (scout) scout_rec(it + 2);
        // ---- level 16, z, and level 32, z: slabs y = warp and warp + 16
#pragma unroll 1
        for (int r = 0; r < 2; ++r) {
            const int y = warp + 16 * r;
            const uint32_t slab = kMain + y * kPlane, q = smem_u32(sm) + slab + (lane >> 4) * 2048;
            const unsigned kb = r ? kz[1] : kz[0];
            const int e = r ? ex[1] : ex[0];
            float v[32];
            unpack16<0>(q + (e & 0xffff) * 4, kb & 0xffffu, v);
            unpack16<16>(q + 1024 + (e >> 16) * 4, kb >> 16, v);
            if (r == 0) {
                float u[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) u[j] = at(sm, corner(lane & 15, y, j));
                line_inv<16, KIND>(u);
                if (lane < 16) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = u[j];
                }
            }
            __syncwarp();
            line_inv<32, KIND>(v);
#pragma unroll
            for (int j = 0; j < 32; ++j) at(sm, slab + j * 128 + lane * 4) = v[j];
        }
        __syncthreads();
        if (scout) find(it + 2, s_off, s_len, s_nb, s_hole, s_src);
        // ---- level 32, y then x: planes z = warp and warp + 16, then straight
        // to the field (copy_to, WaveletCompressor.h:73-82)
        DiffAcc acc;
#pragma unroll 1
        for (int r = 0; r < 2; ++r) {
            const int z = warp + 16 * r;
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = at(sm, kMain + j * kPlane + z * 128 + lane * 4);
            line_inv<32, KIND>(v);
            if (lane == 0) tma_store_wait_read();
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; ++j) at(slot, col_at(lane, j)) = v[j];
            __syncwarp();
            ld_row(slot, lane, v);
            line_inv<32, KIND>(v);
            st_row(slot, lane, v);
            fence_async_smem();
            __syncwarp();
            if (lane == 0) tma_store_3d(fs.list ? fs.maps + cur.field : &fs.map, cur.x, cur.y, cur.z + z, smem_u32(slot));
            if (DIFF) {
                // a lane reads its row 16 bytes at a time: the line must stay in L1
                // between the reads (as streaming loads: 1.42 instead of 1.17 ms at 512^3)
                const CzField &f = fs.list ? fs.list[cur.field] : fs.one;
                const float4 *rr = reinterpret_cast<const float4 *>(
                    diff_ref + ((size_t)(cur.z + z) * f.ny + (size_t)(cur.y + lane)) * f.nx + (size_t)cur.x);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float4 q = __ldg(rr + k);
                    acc.put(v[4 * k], q.x);
                    acc.put(v[4 * k + 1], q.y);
                    acc.put(v[4 * k + 2], q.z);
                    acc.put(v[4 * k + 3], q.w);
                }
            }
        }
        if (DIFF) {
            // block totals in binary64: maxima exact, sums of the compensated
            // partials; order of the record: {e_inf, n_inf, e_1, e_2, n_1, n_2,
            // min, max}, the first two and the last two as maxima
            double(*red)[8] = reinterpret_cast<double(*)[8]>(sm + kRing + kStores * kPlane);
            const double m = warp_fold4(fabs((double)acc.es + acc.ee), (double)acc.ninf, -(double)acc.mn, (double)acc.mx,
                                        [](double a, double b) { return fmax(a, b); });
            const double u = warp_fold4((double)acc.s[0] + (double)acc.c[0], (double)acc.s[1] + (double)acc.c[1],
                                        (double)acc.s[2] + (double)acc.c[2], (double)acc.s[3] + (double)acc.c[3],
                                        [](double a, double b) { return a + b; });
            if ((lane & 7) == 0) {
                const int k = lane >> 3;
                red[warp][k < 2 ? k : k + 4] = k == 2 ? -m : m;
                red[warp][2 + k] = u;
            }
            __syncthreads();
            if (lane == 0 && warp < 8) {  // a warp per quantity: one chain of binary64 operations each
                double r = red[0][warp];
#pragma unroll
                for (int w = 1; w < kNW; ++w) r = diff_fold(warp, r, red[w][warp]);
                diff_out[g * 8 + warp] = r;
            }
        }
    }
    if (lane == 0) tma_store_wait_all();
}

// Totals over blocks, in block order: {e_inf, n_inf, e_1, e_2, n_1, n_2, min, max}.
// Field totals of the per-block statistics, in a fixed order: thread group j
// (of kDiffGroups) folds blocks j, j + kDiffGroups, ... in turn (four loads
// in flight, folded in block order), then the groups fold in order j = 0, 1,
// ... Deterministic for a given block count.
constexpr int kDiffGroups = 128;
__global__ void __launch_bounds__(8 * kDiffGroups)
diff_total_kernel(const double *per_block, long long nblocks, double *total)
{
    __shared__ double part[kDiffGroups][8];
    const int k = threadIdx.x & 7, j = threadIdx.x >> 3;
    double r = 0.0;
    long long g = j;
    if (g < nblocks) {
        r = per_block[g * 8 + k];
        g += kDiffGroups;
    }
    for (; g + 3 * kDiffGroups < nblocks; g += 4 * kDiffGroups) {
        const double x0 = per_block[g * 8 + k], x1 = per_block[(g + kDiffGroups) * 8 + k];
        const double x2 = per_block[(g + 2 * kDiffGroups) * 8 + k], x3 = per_block[(g + 3 * kDiffGroups) * 8 + k];
        r = diff_fold(k, diff_fold(k, diff_fold(k, diff_fold(k, r, x0), x1), x2), x3);
    }
    for (; g < nblocks; g += kDiffGroups) r = diff_fold(k, r, per_block[g * 8 + k]);
    part[j][k] = r;
    __syncthreads();
    // one chain of binary64 operations per quantity, each in a warp of its own
    // (in one warp the three kinds ran one after the other: 22 us a launch)
    if ((threadIdx.x & 31) == 0 && threadIdx.x < 8 * 32) {
        const int q = threadIdx.x >> 5, n = nblocks < kDiffGroups ? (int)nblocks : kDiffGroups;
        double t = part[0][q];
#pragma unroll 8
        for (int i = 1; i < n; ++i) t = diff_fold(q, t, part[i][q]);
        total[q] = t;
    }
}

}  // namespace cz

using namespace cz;

bool cz_field_map(const CzField &f, CUtensorMap *map)
{
    CzEncodeTiled enc = cz_encode_tiled();
    if (!enc) return false;
    // one z plane of a block per box
    const cuuint64_t dim[3] = {(cuuint64_t)f.nx, (cuuint64_t)f.ny, (cuuint64_t)f.nz};
    const cuuint64_t stride[2] = {(cuuint64_t)f.nx * 4, (cuuint64_t)f.nx * f.ny * 4};
    const cuuint32_t box[3] = {32, 32, 1}, es[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(f.data), dim, stride, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t cz_launch_encode(int wtype, const CzFields &fields, long long total_blocks, int zerobits, int shuffle,
                             uint8_t *stage, int *rec_bytes, unsigned long long *queue, int grid, cudaStream_t st,
                             int *err, int variant, CzChunks chunks)
{
    auto launch = [&](auto k) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCodecSmem);
        if (e != cudaSuccess) return e;
        k<<<grid, kNT, kCodecSmem, st>>>(fields, total_blocks, zerobits, shuffle, stage, rec_bytes, queue, err, chunks);
        return cudaGetLastError();
    };
    switch (wkind(wtype)) {
    case 1:
        return launch(variant == 1 ? encode_kernel<1, false> : encode_kernel<1, true>);
    case 2:
        return launch(variant == 1 ? encode_kernel<2, false> : encode_kernel<2, true>);
    default:
        return launch(variant == 1 ? encode_kernel<3, false> : encode_kernel<3, true>);
    }
}

cudaError_t cz_launch_decode(int wtype, const CzFields &fields, long long total_blocks, int shuffle, CzRecords recs,
                             int *flag, unsigned long long *queue, int grid, cudaStream_t st, const float *diff_ref,
                             double *diff_out, CzPlanes planes)
{
    auto launch = [&](auto k) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCodecSmem);
        if (e != cudaSuccess) return e;
        k<<<grid, kNT, kCodecSmem, st>>>(fields, total_blocks, shuffle, recs, flag, queue, diff_ref, diff_out, planes);
        return cudaGetLastError();
    };
    switch (wkind(wtype)) {
    case 1:
        return launch(diff_ref ? decode_kernel<1, true> : decode_kernel<1, false>);
    case 2:
        return launch(diff_ref ? decode_kernel<2, true> : decode_kernel<2, false>);
    default:
        return launch(diff_ref ? decode_kernel<3, true> : decode_kernel<3, false>);
    }
}

cudaError_t cz_launch_diff_total(const double *per_block, long long nblocks, double *total, cudaStream_t st)
{
    if (nblocks < 1) return cudaErrorInvalidValue;
    diff_total_kernel<<<1, 8 * kDiffGroups, 0, st>>>(per_block, nblocks, total);
    return cudaGetLastError();
}
