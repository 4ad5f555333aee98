// Baseline JPEG on sm_100a after the entropy decoder: dequantise + 8x8 integer IDCT, chroma upsampling + YCbCr->RGB.  Second
// half of the zune-jpeg decode datago reaches through image::load_from_memory (src/worker_wds.rs:45) /
// ImageReader::decode (src/worker_files.rs:14-16).
//
// All of it is integer / byte work bound by instruction issue or HBM traffic; no tensor cores.
#include <cstdint>
#include <mutex>

#include "kernels.h"

namespace dg {

// ---------------------------------------------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t owner_of(const OwnerMap& m, uint32_t idx) {
    uint32_t o = __ldg(m.coarse + (idx >> m.shift));
    while (o + 1 < m.n && __ldg(m.first + o + 1) <= idx) ++o;
    return o;
}

// ---------------------------------------------------------------------------------------------------------------
// K2  dequantise + 8x8 inverse DCT (the 13-bit fixed-point "islow" factorisation: columns, round to 2 fractional
//     bits, rows, round, +128, clamp) for every block of a wave, written to 8-bit component planes.
//
//     The stage is bound by integer instruction issue, not by HBM, so the kernel is built to execute few
//     instructions: one thread per block (no exchange between lanes), dequantisation and 16-bit unpacking in one
//     dp2a per coefficient, rounding constants folded into the even part of each butterfly, saturating pack
//     instructions, a reduced butterfly when every block of the warp keeps its energy in the top-left 4x4, and a
//     constant fill when every block of the warp has nothing but a DC term.
//     All arithmetic is exact in 32-bit integers, so regrouping the butterflies cannot change a result.
// ---------------------------------------------------------------------------------------------------------------
constexpr int32_t F_0_298 = 2446, F_0_390 = 3196, F_0_541 = 4433, F_0_765 = 6270, F_0_899 = 7373, F_1_175 = 9633,
                  F_1_501 = 12299, F_1_847 = 15137, F_1_961 = 16069, F_2_053 = 16819, F_2_562 = 20995, F_3_072 = 25172;

// o[k] = (butterfly(x)[k] + RND) >> SHIFT
template <int32_t RND, int SHIFT>
__device__ __forceinline__ void idct8(int32_t x0, int32_t x1, int32_t x2, int32_t x3, int32_t x4, int32_t x5, int32_t x6,
                                      int32_t x7, int32_t (&o)[8]) {
    const int32_t z1e = (x2 + x6) * F_0_541;
    const int32_t t2 = z1e - x6 * F_1_847, t3 = z1e + x2 * F_0_765;
    const int32_t t0 = (x0 + x4) * 8192 + RND, t1 = (x0 - x4) * 8192 + RND;
    const int32_t t10 = t0 + t3, t13 = t0 - t3, t11 = t1 + t2, t12 = t1 - t2;
    int32_t z1 = x7 + x1, z2 = x5 + x3, z3 = x7 + x3, z4 = x5 + x1;
    const int32_t z5 = (z3 + z4) * F_1_175;
    z3 = z5 - z3 * F_1_961;
    z4 = z5 - z4 * F_0_390;
    z1 *= -F_0_899;
    z2 *= -F_2_562;
    const int32_t o0 = x7 * F_0_298 + z1 + z3, o1 = x5 * F_2_053 + z2 + z4, o2 = x3 * F_3_072 + z2 + z3,
                  o3 = x1 * F_1_501 + z1 + z4;
    o[0] = (t10 + o3) >> SHIFT; o[7] = (t10 - o3) >> SHIFT; o[1] = (t11 + o2) >> SHIFT; o[6] = (t11 - o2) >> SHIFT;
    o[2] = (t12 + o1) >> SHIFT; o[5] = (t12 - o1) >> SHIFT; o[3] = (t13 + o0) >> SHIFT; o[4] = (t13 - o0) >> SHIFT;
}

// The same butterfly with x4 = x5 = x6 = x7 = 0 (constants merged; exact because the arithmetic is a ring).
template <int32_t RND, int SHIFT>
__device__ __forceinline__ void idct8_lo4(int32_t x0, int32_t x1, int32_t x2, int32_t x3, int32_t (&o)[8]) {
    const int32_t t2 = x2 * F_0_541, t3 = x2 * (F_0_541 + F_0_765);
    const int32_t t0 = x0 * 8192 + RND;
    const int32_t t10 = t0 + t3, t13 = t0 - t3, t11 = t0 + t2, t12 = t0 - t2;
    const int32_t o0 = x1 * (F_1_175 - F_0_899) + x3 * (F_1_175 - F_1_961);
    const int32_t o1 = x1 * (F_1_175 - F_0_390) + x3 * (F_1_175 - F_2_562);
    const int32_t o2 = x1 * F_1_175 + x3 * (F_3_072 - F_2_562 - F_1_961 + F_1_175);
    const int32_t o3 = x1 * (F_1_501 - F_0_899 - F_0_390 + F_1_175) + x3 * F_1_175;
    o[0] = (t10 + o3) >> SHIFT; o[7] = (t10 - o3) >> SHIFT; o[1] = (t11 + o2) >> SHIFT; o[6] = (t11 - o2) >> SHIFT;
    o[2] = (t12 + o1) >> SHIFT; o[5] = (t12 - o1) >> SHIFT; o[3] = (t13 + o0) >> SHIFT; o[4] = (t13 - o0) >> SHIFT;
}

// ... and with x2 = x3 = 0 as well.
template <int32_t RND, int SHIFT>
__device__ __forceinline__ void idct8_lo2(int32_t x0, int32_t x1, int32_t (&o)[8]) {
    const int32_t t0 = x0 * 8192 + RND;
    const int32_t o0 = x1 * (F_1_175 - F_0_899), o1 = x1 * (F_1_175 - F_0_390), o2 = x1 * F_1_175,
                  o3 = x1 * (F_1_501 - F_0_899 - F_0_390 + F_1_175);
    o[0] = (t0 + o3) >> SHIFT; o[7] = (t0 - o3) >> SHIFT; o[1] = (t0 + o2) >> SHIFT; o[6] = (t0 - o2) >> SHIFT;
    o[2] = (t0 + o1) >> SHIFT; o[5] = (t0 - o1) >> SHIFT; o[3] = (t0 + o0) >> SHIFT; o[4] = (t0 - o0) >> SHIFT;
}

// packs sat_u8 of four ints into one word, first argument in the lowest byte
__device__ __forceinline__ uint32_t pack_sat_u8(int32_t a, int32_t b, int32_t c, int32_t d) {
    uint32_t hi, r;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
    return r;
}

// coefficient pair (low half, high half of cw) times the two quantisers in bytes 0 and 3 of qw
__device__ __forceinline__ void dequant_pair(uint32_t cw, uint32_t qw, int32_t& lo, int32_t& hi) {
    asm("dp2a.lo.s32.u32 %0, %1, %2, 0;" : "=r"(lo) : "r"(cw), "r"(qw));
    asm("dp2a.hi.s32.u32 %0, %1, %2, 0;" : "=r"(hi) : "r"(cw), "r"(qw));
}

constexpr int32_t kRound1 = 1 << 10, kRound2 = (1 << 17) + (128 << 18);
constexpr int kIdctThreads = 128;

// The rows of a staged block (32 blocks of a warp, row r of block b at chunk b * 8 + (r ^ (b & 7))) that its class covers;
// the others are zero and were not fetched.  The DC term comes from info[].
__device__ __forceinline__ void read_block(const uint4* rows, uint32_t swz, uint32_t nrows, uint32_t dc, uint4 (&c)[8]) {
#pragma unroll
    for (int r = 0; r < 8; ++r) c[r] = (uint32_t)r < nrows ? rows[r ^ swz] : make_uint4(0, 0, 0, 0);
    c[0].x = (c[0].x & 0xFFFF0000u) | (dc & 0xFFFFu);
}

// Dequantise + inverse DCT of the calling lane's block; c = its coefficient rows (only the part class `cls` covers is
// read), qq = the quantiser rows in the dp2a layout.  emit(r, lo, hi) receives row r of the result as two words of
// four saturated samples.  cls must be the same for all lanes of the warp and no sparser than any lane's block.
template <class Emit>
__device__ __forceinline__ void idct_block(const uint4 (&c)[8], const uint4* __restrict__ qq, int cls, Emit&& emit) {
    if (cls == kClsDc) {
        // flat blocks: both passes reduce to shifts of the DC term
        int32_t lo, hi;
        dequant_pair(c[0].x, __ldg(reinterpret_cast<const uint32_t*>(qq)), lo, hi);
        const int32_t wsv = (lo * 8192 + kRound1) >> 11;
        const int32_t v = (wsv * 8192 + kRound2) >> 18;
        const uint32_t px4 = pack_sat_u8(v, v, v, v);
#pragma unroll
        for (int r = 0; r < 8; ++r) emit(r, px4, px4);
    } else if (cls == kCls2x2) {
        int32_t x[2][2], ws[8][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) dequant_pair(c[r].x, __ldg(reinterpret_cast<const uint32_t*>(qq + r)), x[r][0], x[r][1]);
#pragma unroll
        for (int col = 0; col < 2; ++col) {
            int32_t o[8];
            idct8_lo2<kRound1, 11>(x[0][col], x[1][col], o);
#pragma unroll
            for (int r = 0; r < 8; ++r) ws[r][col] = o[r];
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            int32_t o[8];
            idct8_lo2<kRound2, 18>(ws[r][0], ws[r][1], o);
            emit(r, pack_sat_u8(o[0], o[1], o[2], o[3]), pack_sat_u8(o[4], o[5], o[6], o[7]));
        }
    } else if (cls == kCls4x4) {
        int32_t x[4][4], ws[8][4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint2 qv = __ldg(reinterpret_cast<const uint2*>(qq + r));
            dequant_pair(c[r].x, qv.x, x[r][0], x[r][1]);
            dequant_pair(c[r].y, qv.y, x[r][2], x[r][3]);
        }
#pragma unroll
        for (int col = 0; col < 4; ++col) {
            int32_t o[8];
            idct8_lo4<kRound1, 11>(x[0][col], x[1][col], x[2][col], x[3][col], o);
#pragma unroll
            for (int r = 0; r < 8; ++r) ws[r][col] = o[r];
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            int32_t o[8];
            idct8_lo4<kRound2, 18>(ws[r][0], ws[r][1], ws[r][2], ws[r][3], o);
            emit(r, pack_sat_u8(o[0], o[1], o[2], o[3]), pack_sat_u8(o[4], o[5], o[6], o[7]));
        }
    } else {
        int32_t ws[8][8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const uint4 qv = __ldg(qq + r);
            dequant_pair(c[r].x, qv.x, ws[r][0], ws[r][1]);
            dequant_pair(c[r].y, qv.y, ws[r][2], ws[r][3]);
            dequant_pair(c[r].z, qv.z, ws[r][4], ws[r][5]);
            dequant_pair(c[r].w, qv.w, ws[r][6], ws[r][7]);
        }
#pragma unroll
        for (int col = 0; col < 8; ++col) {
            int32_t o[8];
            idct8<kRound1, 11>(ws[0][col], ws[1][col], ws[2][col], ws[3][col], ws[4][col], ws[5][col], ws[6][col], ws[7][col], o);
#pragma unroll
            for (int r = 0; r < 8; ++r) ws[r][col] = o[r];
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            int32_t o[8];
            idct8<kRound2, 18>(ws[r][0], ws[r][1], ws[r][2], ws[r][3], ws[r][4], ws[r][5], ws[r][6], ws[r][7], o);
            emit(r, pack_sat_u8(o[0], o[1], o[2], o[3]), pack_sat_u8(o[4], o[5], o[6], o[7]));
        }
    }
}

// the class a whole warp can run: the least sparse of its lanes' classes
__device__ __forceinline__ int warp_class(int cls) { return (int)__reduce_min_sync(0xFFFFFFFFu, (unsigned)cls); }

#ifndef DG_IDCT_MIN_CTAS
#define DG_IDCT_MIN_CTAS 7
#endif
__global__ void __launch_bounds__(kIdctThreads, DG_IDCT_MIN_CTAS) k_idct(JpegWave w, uint32_t first, uint32_t count) {
    const uint32_t local = blockIdx.x * kIdctThreads + threadIdx.x;
    const uint32_t g = first + min(local, count - 1);
    // A warp's 32 blocks are 4 KB of consecutive coefficients.  The rows their classes cover are fetched with coalesced
    // 16-byte asynchronous copies into shared memory (one chunk = one block row) while the descriptor look-ups run; then
    // every lane reads back the rows of its own block.  Row r of block b sits at chunk b * 8 + (r ^ (b & 7)): copy-in and
    // read-back both touch eight different 16-byte bank groups per quarter warp.
    // (One 16-byte load per lane and row straight from global memory makes every instruction touch 32 lines.)
    __shared__ __align__(16) uint4 s_coef[kIdctThreads / 32][256];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t img = owner_of(w.blocks, g);
    const JpegDesc& d = w.descs[img];
    let_next_start();
    wait_for_previous();
    const uint32_t v = w.info[g];
    const int cls = (int)((v >> 16) & 3u);
    const uint32_t nrows = class_rows(cls);
    {
        const uint32_t warp_first = blockIdx.x * kIdctThreads + warp * 32;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bb = i * 4 + (lane >> 3), r = lane & 7;
            const uint32_t gb = first + min(warp_first + bb, count - 1);
            if (r < __shfl_sync(0xFFFFFFFFu, nrows, bb)) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_coef[warp][bb * 8 + (r ^ (bb & 7))]);
                const void* src = w.coef + (size_t)gb * 64 + r * 8;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const uint32_t blk = g - (uint32_t)d.block_off;
    const bool valid = local < count && blk < d.nblocks;  // (images start at multiples of eight blocks)
    const uint32_t mcu = blk / d.bpm, k = blk - mcu * d.bpm;
    const uint32_t my = mcu / d.mcux, mx = mcu - my * d.mcux;
    const uint32_t luma = d.hs * d.vs;
    uint32_t comp, bx, by;
    if (k < luma) { comp = 0; const uint32_t ky = k / d.hs; bx = mx * d.hs + (k - ky * d.hs); by = my * d.vs + ky; }
    else { comp = k - luma + 1; bx = mx; by = my; }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    uint4 c[8];
    read_block(&s_coef[warp][lane * 8], lane & 7, nrows, v, c);
    const uint4* qq = reinterpret_cast<const uint4*>(w.qt32 + (size_t)d.qt[comp] * 32);
    uint8_t* dst = w.planes + d.plane_off[comp] + (size_t)(by * 8) * d.plane_pitch[comp] + bx * 8;
    const uint32_t pitch = d.plane_pitch[comp];
    idct_block(c, qq, warp_class(cls), [&](int r, uint32_t lo, uint32_t hi) {
        if (valid) *reinterpret_cast<uint2*>(dst + (size_t)r * pitch) = make_uint2(lo, hi);
    });
}

void launch_idct(const JpegWave& w, uint32_t first, uint32_t count, cudaStream_t s) {
    if (count) launch_after(k_idct, (count + kIdctThreads - 1) / kIdctThreads, kIdctThreads, 0, s, w, first, count);
}

// ---------------------------------------------------------------------------------------------------------------
// K3  chroma upsampling + YCbCr -> RGB (16-bit fixed point constants 1.402, 0.34414, 0.71414, 1.772), interleaved
//     RGB8 out.  A CTA owns 256 pixels of four MCU rows, a thread 8 pixels of every eighth row of the tile.
//       4:2:0  triangle filter: every output sample is (9a + 3b + 3c + d + bias) >> 4 over its 2x2 chroma
//              neighbourhood -- one dp4a on bytes gathered from a shared-memory tile (1-sample halo, clamped to the
//              real plane extent, which is what the edge rules of the filter amount to);
//       4:4:4  and grayscale: straight from the planes;
//       4:2:2  triangle filter along the row, from the planes;
//       other samplings and chroma planes at most two samples wide: a plain per-pixel path.
//     The +128 offsets and the rounding term are folded into one constant per channel; the luma byte is added with a
//     one-hot dp4a; results are saturated and packed four at a time.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kColorThreads = 256;
constexpr int kCTileCols = kColorTileW / 2 + 8;  // 4 bytes of left margin (halo in the last one), halo + slack right

__device__ __forceinline__ uint32_t dp4a_u(uint32_t a, uint32_t b, uint32_t c) { return __dp4a(a, b, c); }

// The four bytes (cb, cb, cr, cr), each minus 128, of the pixel whose samples are byte `at` of cb and of cr.
template <uint32_t AT> __device__ __forceinline__ uint32_t chroma_word(uint32_t cb, uint32_t cr) { return __byte_perm(cb, cr, AT | AT << 4 | (4 + AT) << 8 | (4 + AT) << 12); }

// 8 pixels: luma words y0, y1; chroma words; out: 24 bytes.
// R = Y + ((91881 * (cr - 128) + 32768) >> 16) = (91881 * (cr - 128) + ((Y << 16) + 32768)) >> 16, and likewise for G and
// B: the luma byte is moved into bits 16..23 of a word that already carries the rounding term (one byte permute per pixel).
// The 17-bit constants are applied as two halves to a sample that is in the word twice (dp2a), so that no sample has to be
// taken out of its word; results are taken from the upper halves two at a time and clamped together.  That leaves the
// integer pipe, which bounds the colour kernels, 5.8 instructions per pixel instead of 7.5 with a shift per sample and per
// channel, and the chroma filters one less.
__device__ __forceinline__ void ycc_to_rgb8(uint32_t y0, uint32_t y1, const uint32_t (&c)[8], uint32_t (&out)[6]) {
    constexpr uint32_t kR = 45940u | 45941u << 16, kB = 58065u | 58065u << 16;                              // 91881, 116130
    constexpr uint32_t kGb = (uint32_t)(uint16_t)-11277 * 0x10001u, kGr = (uint32_t)(uint16_t)-23401 * 0x10001u;  // -22554, -46802
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // four pixels at a time keeps fewer values live
        const uint32_t yw = h ? y1 : y0;
        uint32_t v[12];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t y16 = __byte_perm(yw, 0x00008000u, 0x7054u | ((uint32_t)i << 8)), w = c[4 * h + i];  // 0x00YY8000
            asm("dp2a.hi.u32.s32 %0, %1, %2, %3;" : "=r"(v[3 * i]) : "r"(kR), "r"(w), "r"(y16));
            asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(v[3 * i + 1]) : "r"(kGb), "r"(w), "r"(y16));
            asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(v[3 * i + 1]) : "r"(kGr), "r"(w), "r"(v[3 * i + 1]));
            asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(v[3 * i + 2]) : "r"(kB), "r"(w), "r"(y16));
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const uint32_t lo = __vimin_s16x2_relu(__byte_perm(v[4 * j], v[4 * j + 1], 0x7632), 0x00FF00FFu);
            const uint32_t hi = __vimin_s16x2_relu(__byte_perm(v[4 * j + 2], v[4 * j + 3], 0x7632), 0x00FF00FFu);
            out[3 * h + j] = __byte_perm(lo, hi, 0x6420);
        }
    }
}

// The lanes of `lanes` (lane 0 and its neighbours up, called by all of them together) store the 24 bytes of eight pixels each,
// at consecutive places of a row.  Rows of odd-sized images start at any byte: a lane then stores the words that begin in
// its piece, the first of them with the last bytes of its left neighbour's; the ends of the run go byte by byte (a byte at
// a time for all of it, as before: 503 us for 96 images of 0.6 Mpixel, 141 by words).  npx < 8: the ragged piece at the right edge.
__device__ __forceinline__ void store_rgb8(uint8_t* o, const uint32_t (&px)[6], int npx, uint32_t lanes) {
    const uint32_t m = (uint32_t)(reinterpret_cast<uintptr_t>(o) & 7u);  // the same for all lanes
    if (m == 0) {
        if (npx == 8) {
            uint2* o2 = reinterpret_cast<uint2*>(o);
            __stcs(o2, make_uint2(px[0], px[1])); __stcs(o2 + 1, make_uint2(px[2], px[3])); __stcs(o2 + 2, make_uint2(px[4], px[5]));
            return;
        }
    } else {
        const uint32_t lane = threadIdx.x & 31, before = __shfl_up_sync(lanes, px[5], 1), right = __shfl_down_sync(lanes, (uint32_t)npx, 1);
        if (npx == 8) {
            const uint32_t k = m & 3u, sh = (32u - 8u * k) & 31u;
            uint32_t* w = reinterpret_cast<uint32_t*>(o - k);
            if (k == 0) {
#pragma unroll
                for (int i = 0; i < 6; ++i) __stcs(w + i, px[i]);
                return;
            }
            if (lane) __stcs(w, __funnelshift_r(before, px[0], sh));
            else
                for (uint32_t i = 0; i < 4 - k; ++i) o[i] = (uint8_t)(px[0] >> (8 * i));
#pragma unroll
            for (int i = 1; i < 6; ++i) __stcs(w + i, __funnelshift_r(px[i - 1], px[i], sh));
            const bool last = lane == 31 || !((lanes >> (lane + 1)) & 1u) || right != 8;  // nobody else stores this piece's last bytes
            if (last)
                for (uint32_t i = 4 - k; i < 4; ++i) o[20 + i] = (uint8_t)(px[5] >> (8 * i));
            return;
        }
    }
    // ragged right edge: byte by byte, the word index resolved at compile time
    const int nb = npx * 3;
#pragma unroll
    for (int wi = 0; wi < 6; ++wi)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (wi * 4 + k < nb) o[wi * 4 + k] = (uint8_t)(px[wi] >> (8 * k));
}

struct ChromaPlane {  // per-pixel path
    const uint8_t* p;
    uint32_t pitch;
    int dh, hs, vs;
    __device__ __forceinline__ int px(int x, int y) const { return (int)load_global(p + (size_t)y * pitch + x); }
    __device__ __forceinline__ int at(int x, int y) const {
        if (hs == 2) return px(x >> 1, vs == 2 ? y >> 1 : y);  // planes at most two samples wide: replicated
        const int cy = y >> 1, far = min(max((y & 1) ? cy + 1 : cy - 1, 0), dh - 1);  // 4:4:0: triangle filter down the column
        return (3 * px(x, cy) + px(x, far) + ((y & 1) ? 2 : 1)) >> 2;
    }
};

constexpr int kCTileRows = 8 * (int)kColorMcuRows + 2;  // chroma rows of a 4:2:0 tile plus one halo row above and below

// Chroma tile of a 4:2:0 image: rows cy0-1 .. cy0+32, columns cx0-4 .. cx0+131 as aligned words; s_c column = chroma column
// - cx0 + 4.  Coordinates are clamped to the real plane extent (dw x dh samples) and the first / last real column is
// replicated into the halo position, which is what the edge rules of the triangle filter amount to.
// Warp q loads tile rows q, q + 8, ... of both components; a lane loads word `lane` and, for two lanes, word 32 + lane.
// Two steps, both by every thread of the CTA (256), with a __syncthreads() after each: chroma_tile_fetch, chroma_tile_edges.
template <int ROWS>
__device__ __forceinline__ void chroma_tile_fetch(uint8_t (&s_c)[2][ROWS][kCTileCols], const uint8_t* planes, const JpegDesc& d,
                                                  int tx, int ty, int dh) {
    constexpr int kCTileRows = ROWS;
    const int lane = threadIdx.x & 31, rowi = threadIdx.x >> 5;
    const int cx0 = tx * (int)(kColorTileW / 2), cy0 = ty * 8 * (int)kColorMcuRows;
    constexpr int kWords = kCTileCols / 4;  // 34
    const uint32_t cpitch = d.plane_pitch[1];
    const int wmax = (int)(cpitch / 4) - 1, w0 = cx0 / 4 - 1;
    const uint8_t* cb_base = planes + d.plane_off[1];
    const uint8_t* cr_base = planes + d.plane_off[2];
#pragma unroll
    for (int rr = 0; rr < (kCTileRows + 7) / 8; ++rr) {
        const int r = rowi + 8 * rr;
        if (r < kCTileRows) {
            const int gy = min(max(cy0 + r - 1, 0), dh - 1);
            const uint32_t* gb = reinterpret_cast<const uint32_t*>(cb_base + (size_t)gy * cpitch);
            const uint32_t* gr = reinterpret_cast<const uint32_t*>(cr_base + (size_t)gy * cpitch);
            uint32_t* sb = reinterpret_cast<uint32_t*>(s_c[0][r]);
            uint32_t* sr = reinterpret_cast<uint32_t*>(s_c[1][r]);
            const int g0 = min(max(w0 + lane, 0), wmax);
            sb[lane] = load_global(gb + g0);
            sr[lane] = load_global(gr + g0);
            if (lane < kWords - 32) {
                const int g1 = min(max(w0 + 32 + lane, 0), wmax);
                sb[32 + lane] = load_global(gb + g1);
                sr[32 + lane] = load_global(gr + g1);
            }
        }
    }
}

template <int ROWS>
__device__ __forceinline__ void chroma_tile_edges(uint8_t (&s_c)[2][ROWS][kCTileCols], int tx, int dw) {
    constexpr int kCTileRows = ROWS;
    const int cx0 = tx * (int)(kColorTileW / 2);
    if (threadIdx.x < 2 * kCTileRows) {
        const int comp = threadIdx.x / kCTileRows, r = threadIdx.x - comp * kCTileRows;
        if (cx0 == 0) s_c[comp][r][3] = s_c[comp][r][4];
        const int last = dw - 1 - cx0;  // tile-local index of the last real column
        if (last >= 0 && last < (int)(kColorTileW / 2)) s_c[comp][r][4 + last + 1] = s_c[comp][r][4 + last];
    }
}

__device__ __forceinline__ void load_chroma_tile(uint8_t (&s_c)[2][kCTileRows][kCTileCols], const uint8_t* planes, const JpegDesc& d,
                                                 int tx, int ty, int dw, int dh) {
    chroma_tile_fetch(s_c, planes, d, tx, ty, dh);
    __syncthreads();
    chroma_tile_edges(s_c, tx, dw);
    __syncthreads();
}

// Triangle upsampling of the chroma for 8 pixels of two output rows that read the same two chroma rows: row A has
// tile row p as its near row and p + 1 as its far row, row B the other way round (output rows 2j+1 and 2j+2 of the
// image).  cl = s_c column of the thread's first chroma sample (a word boundary).  a, b: the pixels' chroma words.
template <int ROWS = kCTileRows>
__device__ __forceinline__ void chroma_pair(const uint8_t (&s_c)[2][ROWS][kCTileCols], int p, int cl, uint32_t (&a)[8], uint32_t (&b)[8]) {
    // sixteen times the weights 9, 3, 3, 1 (and of the rounding term minus 128): the sample is byte 1 of the result
    constexpr uint32_t kEvenA = 0x30901030u, kOddA = 0x10303090u;  // bytes: (near a, far a, near b, far b)
    constexpr uint32_t kEvenB = 0x90303010u, kOddB = 0x30109030u;  // the same bytes with near and far exchanged
    constexpr uint32_t kE = (uint32_t)((8 - 2048) * 16), kO = (uint32_t)((7 - 2048) * 16);
    uint32_t va[2][8], vb[2][8];
#pragma unroll
    for (int comp = 0; comp < 2; ++comp) {
        const uint32_t* nr = reinterpret_cast<const uint32_t*>(&s_c[comp][p][cl]);
        const uint32_t* fr = reinterpret_cast<const uint32_t*>(&s_c[comp][p + 1][cl]);
        const uint32_t Ln = nr[-1], Mn = nr[0], Nn = nr[1], Lf = fr[-1], Mf = fr[0], Nf = fr[1];
        const uint32_t I0 = __byte_perm(Mn, Mf, 0x5140), J = __byte_perm(Mn, Mf, 0x6251), I1 = __byte_perm(Mn, Mf, 0x7362);
        const uint32_t Lp = __byte_perm(__byte_perm(Ln, Lf, 0x0073), I0, 0x5410);  // (c-1, c)
        const uint32_t Rp = __byte_perm(I1, __byte_perm(Nn, Nf, 0x0040), 0x5432);  // (c+3, c+4)
        const uint32_t even[4] = {Lp, I0, J, I1}, odd[4] = {I0, J, I1, Rp};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            va[comp][2 * i] = dp4a_u(even[i], kEvenA, kE); va[comp][2 * i + 1] = dp4a_u(odd[i], kOddA, kO);
            vb[comp][2 * i] = dp4a_u(even[i], kEvenB, kE); vb[comp][2 * i + 1] = dp4a_u(odd[i], kOddB, kO);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) { a[i] = chroma_word<1>(va[0][i], va[1][i]); b[i] = chroma_word<1>(vb[0][i], vb[1][i]); }
}

__global__ void __launch_bounds__(kColorThreads, 4) k_color(JpegWave w, uint32_t first_tile) {
    __shared__ __align__(16) uint8_t s_c[2][kCTileRows][kCTileCols];
    __shared__ uint32_t s_img;
    if (threadIdx.x == 0) s_img = owner_of(w.color_tiles, first_tile + blockIdx.x);
    let_next_start();
    wait_for_previous();
    __syncthreads();
    const uint8_t* const planes = from_previous(w.planes);
    const uint32_t img = s_img;
    const JpegDesc& d = w.descs[img];
    const uint32_t tile = first_tile + blockIdx.x - w.color_tiles.first[img];
    const int W = (int)d.width, H = (int)d.height, hs = (int)d.hs, vs = (int)d.vs;
    const uint32_t tiles_x = (d.width + kColorTileW - 1) / kColorTileW;
    const uint32_t ty = tile / tiles_x, tx = tile - ty * tiles_x;
    const int lane = threadIdx.x & 31, rowi = threadIdx.x >> 5;  // 32 column groups x 8 rows
    const int x = (int)tx * (int)kColorTileW + lane * 8;
    const int y_base = (int)ty * 8 * vs * (int)kColorMcuRows;
    const int nsteps = vs * (int)kColorMcuRows;  // a thread converts rows rowi, rowi + 8, ... of the tile
    uint8_t* out = w.out + d.out_off;
    const uint8_t* yp = planes + d.plane_off[0];
    const uint32_t ypitch = d.plane_pitch[0];

    if (d.ncomp == 1) {  // grayscale: copy the real extent of the luma plane
        if (x >= W) return;
        const int npx = min(8, W - x);
        for (int k = 0; k < nsteps; ++k) {
            const int y = y_base + rowi + 8 * k;
            if (y >= H) break;
            const uint2 v = load_global(reinterpret_cast<const uint2*>(yp + (size_t)y * ypitch + x));
            uint8_t* o = out + (size_t)y * d.out_pitch + x;
            if (npx == 8 && (reinterpret_cast<uintptr_t>(o) & 7u) == 0) __stcs(reinterpret_cast<uint2*>(o), v);
            else for (int i = 0; i < npx; ++i) o[i] = (uint8_t)((i < 4 ? v.x : v.y) >> (8 * (i & 3)));
        }
        return;
    }
    const int dw = (W + hs - 1) / hs, dh = (H + vs - 1) / vs;
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, x < W);
    if (hs == 2 && vs == 2 && dw > 2) {
        load_chroma_tile(s_c, planes, d, (int)tx, (int)ty, dw, dh);
        if (x >= W) return;
        const int cl = lane * 4 + 4;  // s_c column of this thread's first chroma sample (a word boundary)
        const int npx = min(8, W - x);
        // Output rows 2j+1 and 2j+2 read the same two chroma rows (j and j+1) with the near / far weights exchanged, so
        // the tile is shifted up by one row -- it covers rows 64 ty - 1 .. 64 ty + 62 -- and a thread converts such a
        // pair at a time: the byte gathering is done once, the second row only swaps the weights.
        const int y_first = (int)ty * 8 * 2 * (int)kColorMcuRows - 1;
        auto luma = [&](int y) -> uint2 {
            return (y >= 0 && y < H) ? load_global(reinterpret_cast<const uint2*>(yp + (size_t)y * ypitch + x)) : make_uint2(0, 0);
        };
        uint2 nextA = luma(y_first + 2 * rowi), nextB = luma(y_first + 2 * rowi + 1);
#pragma unroll 1
        for (int m = 0; m < (int)kColorMcuRows; ++m) {
            const int p = rowi + 8 * m;  // pair index inside the tile = s_c row of the upper chroma row
            const int yA = y_first + 2 * p, yB = yA + 1;
            if (yA >= H) break;
            const uint2 ya = nextA, yb = nextB;
            if (m + 1 < (int)kColorMcuRows) { nextA = luma(yA + 16); nextB = luma(yB + 16); }  // next pair's luma in flight
            uint32_t a[8], b[8];
            chroma_pair(s_c, p, cl, a, b);
            uint32_t px[6];
            if (yA >= 0) {
                ycc_to_rgb8(ya.x, ya.y, a, px);
                store_rgb8(out + (size_t)yA * d.out_pitch + x * 3, px, npx, lanes);
            }
            if (yB < H) {
                ycc_to_rgb8(yb.x, yb.y, b, px);
                store_rgb8(out + (size_t)yB * d.out_pitch + x * 3, px, npx, lanes);
            }
        }
        return;
    }
    if (x >= W) return;
    const int npx = min(8, W - x);
    if (hs == 1 && vs == 1) {
        for (int k = 0; k < nsteps; ++k) {
            const int y = y_base + rowi + 8 * k;
            if (y >= H) break;
            const uint2 b = load_global(reinterpret_cast<const uint2*>(planes + d.plane_off[1] + (size_t)y * d.plane_pitch[1] + x));
            const uint2 r = load_global(reinterpret_cast<const uint2*>(planes + d.plane_off[2] + (size_t)y * d.plane_pitch[2] + x));
            const uint32_t b0 = b.x ^ 0x80808080u, b1 = b.y ^ 0x80808080u, r0 = r.x ^ 0x80808080u, r1 = r.y ^ 0x80808080u;
            const uint32_t c[8] = {chroma_word<0>(b0, r0), chroma_word<1>(b0, r0), chroma_word<2>(b0, r0), chroma_word<3>(b0, r0),
                                   chroma_word<0>(b1, r1), chroma_word<1>(b1, r1), chroma_word<2>(b1, r1), chroma_word<3>(b1, r1)};
            const uint2 yv = load_global(reinterpret_cast<const uint2*>(yp + (size_t)y * ypitch + x));
            uint32_t px[6];
            ycc_to_rgb8(yv.x, yv.y, c, px);
            store_rgb8(out + (size_t)y * d.out_pitch + x * 3, px, npx, lanes);
        }
        return;
    }
    if (hs == 2 && vs == 1 && dw > 2) {
        // 4:2:2: (3 near + far + 1 or 2) >> 2 along the row.  A thread's eight pixels read four chroma samples (one aligned
        // word) and their two neighbours; samples behind the real extent are the last real one, which makes the general
        // form give the edge rules (3 t + t + 1 or 2) >> 2 = t.
        const int c0 = x >> 1;
        const bool inner = c0 + 4 < dw;
#pragma unroll 2
        for (int k = 0; k < nsteps; ++k) {
            const int y = y_base + rowi + 8 * k;
            if (y >= H) break;
            int32_t cbv[8], crv[8];
#pragma unroll
            for (int comp = 1; comp <= 2; ++comp) {
                const uint8_t* row = planes + d.plane_off[comp] + (size_t)y * d.plane_pitch[comp];
                const uint32_t q = load_global(reinterpret_cast<const uint32_t*>(row + c0));
                int32_t t[6];
                t[0] = (int32_t)load_global(row + max(c0 - 1, 0));
#pragma unroll
                for (int i = 0; i < 4; ++i) t[i + 1] = (int32_t)((q >> (8 * i)) & 255u);
                if (inner) t[5] = (int32_t)load_global(row + c0 + 4);
                else {
                    const int32_t last = (int32_t)load_global(row + dw - 1);
#pragma unroll
                    for (int i = 1; i < 6; ++i) if (c0 + i - 1 >= dw) t[i] = last;
                }
                int32_t (&v)[8] = comp == 1 ? cbv : crv;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    v[2 * i] = ((3 * t[i + 1] + t[i] + 1) >> 2) - 128;
                    v[2 * i + 1] = ((3 * t[i + 1] + t[i + 2] + 2) >> 2) - 128;
                }
            }
            const uint2 yv = load_global(reinterpret_cast<const uint2*>(yp + (size_t)y * ypitch + x));
            uint32_t px[6];
            uint32_t c[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) c[i] = chroma_word<0>((uint32_t)cbv[i], (uint32_t)crv[i]);
            ycc_to_rgb8(yv.x, yv.y, c, px);
            store_rgb8(out + (size_t)y * d.out_pitch + x * 3, px, npx, lanes);
        }
        return;
    }
    // remaining samplings (4:4:0, chroma planes at most two samples wide): one pixel at a time
    const ChromaPlane cbp{planes + d.plane_off[1], d.plane_pitch[1], dh, hs, vs};
    const ChromaPlane crp{planes + d.plane_off[2], d.plane_pitch[2], dh, hs, vs};
#pragma unroll 1
    for (int k = 0; k < nsteps; ++k) {
        const int y = y_base + rowi + 8 * k;
        if (y >= H) break;
#pragma unroll 1
        for (int i = 0; i < npx; ++i) {
            const int Y = (int)load_global(yp + (size_t)y * ypitch + x + i);
            const int cb = cbp.at(x + i, y) - 128, cr = crp.at(x + i, y) - 128;
            uint8_t* o = out + (size_t)y * d.out_pitch + (x + i) * 3;
            o[0] = (uint8_t)min(max(Y + ((91881 * cr + 32768) >> 16), 0), 255);
            o[1] = (uint8_t)min(max(Y + ((-22554 * cb - 46802 * cr + 32768) >> 16), 0), 255);
            o[2] = (uint8_t)min(max(Y + ((116130 * cb + 32768) >> 16), 0), 255);
        }
    }
}

void launch_color(const JpegWave& w, uint32_t first_tile, uint32_t count, cudaStream_t s) {
    if (count) launch_after(k_color, count, kColorThreads, 0, s, w, first_tile);
}

// ---------------------------------------------------------------------------------------------------------------
// Fused path for three-component 4:2:0 images (the common case): the luma samples never go to memory.
//   k_idct_chroma  IDCT of the Cb and Cr blocks only, into the chroma planes (0.5 bytes per pixel instead of 1.5);
//   k_luma_color   one CTA per 256 x 64 pixel tile (16 x 4 MCUs = 256 luma blocks, one per thread): luma coefficients
//                  staged with asynchronous copies, the chroma tile (with its halo, which is why chroma cannot be
//                  reconstructed tile by tile) loaded from the planes meanwhile, luma IDCT into shared memory, then
//                  upsampling and colour conversion from shared memory, RGB out.
// Traffic per pixel, at most (all rows of all blocks): 1 + 0.5 (chroma) + 2 + 0.5 + 3 (fused kernel), against
// 3 + 1.5 + 1.5 + 3 for the two general kernels.
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kIdctThreads, DG_IDCT_MIN_CTAS) k_idct_chroma(JpegWave w, uint32_t first, uint32_t count) {
    const uint32_t local = blockIdx.x * kIdctThreads + threadIdx.x;
    const bool valid = local < count;
    const uint32_t q = first + min(local, count - 1);
    __shared__ __align__(16) uint4 s_coef[kIdctThreads / 32][256];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t o = owner_of(w.fused_chroma, q);
    const JpegDesc& d = w.descs[w.fused_first + o];
    const uint32_t ql = q - __ldg(w.fused_chroma.first + o);
    const uint32_t mcu = ql >> 1, which = ql & 1u;
    const uint32_t blk = (uint32_t)d.block_off + mcu * 6u + 4u + which;  // this lane's block in the coefficient array
    let_next_start();
    wait_for_previous();
    const uint32_t v = w.info[blk];
    const int cls = (int)((v >> 16) & 3u);
    const uint32_t nrows = class_rows(cls);
    // Lanes 2j and 2j + 1 hold the Cb and Cr block of one MCU: 256 consecutive bytes.  Step i copies the rows of blocks
    // 4i .. 4i + 3 of the warp, lane l row l % 8 of block 4i + l / 8 (block addresses come from the owning lanes).
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t bb = i * 4 + (lane >> 3), r = lane & 7;
        const uint32_t gb = __shfl_sync(0xFFFFFFFFu, blk, bb);
        if (r < __shfl_sync(0xFFFFFFFFu, nrows, bb)) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_coef[warp][bb * 8 + (r ^ (bb & 7))]);
            const void* src = w.coef + (size_t)gb * 64 + r * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t my = mcu / d.mcux, mx = mcu - my * d.mcux;
    const uint32_t comp = 1u + which;
    const uint4* qq = reinterpret_cast<const uint4*>(w.qt32 + (size_t)d.qt[comp] * 32);
    const uint32_t pitch = d.plane_pitch[comp];
    uint8_t* dst = w.planes + d.plane_off[comp] + (size_t)(my * 8) * pitch + mx * 8;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    uint4 c[8];
    read_block(&s_coef[warp][lane * 8], lane & 7, nrows, v, c);
    idct_block(c, qq, warp_class(cls), [&](int r, uint32_t lo, uint32_t hi) {
        if (valid) *reinterpret_cast<uint2*>(dst + (size_t)r * pitch) = make_uint2(lo, hi);
    });
}

void launch_idct_chroma(const JpegWave& w, uint32_t first, uint32_t count, cudaStream_t s) {
    if (count) launch_after(k_idct_chroma, (count + kIdctThreads - 1) / kIdctThreads, kIdctThreads, 0, s, w, first, count);
}

constexpr int kFusedThreads = 64 * (int)kFusedMcuRows;
constexpr int kFusedWarps = kFusedThreads / 32;
constexpr int kFTileRows = 8 * (int)kFusedMcuRows + 2;  // chroma rows of a tile plus one halo row above and below
constexpr int kLumaPitch = kColorTileW + 8;  // 8 * pitch = 64 (mod 128): the two block rows a half warp stores to fall into different banks
constexpr int kLumaRows = 16 * (int)kFusedMcuRows;

// What a CTA needs to know about its tile.
struct TileInfo {
    const int16_t* coef;   // first coefficient block of the image
    const uint32_t* info;  // DC term and class of its blocks
    const uint8_t* cb;     // chroma planes
    const uint8_t* cr;
    uint8_t* out;          // decoded image
    const uint4* qq;       // luma quantiser rows (dp2a layout)
    uint32_t mcux, mcuy, width, height, cpitch, tx, ty, opitch;  // opitch: bytes per row of the decoded image
};

struct FusedSmem {
    uint4 coef[kFusedThreads / 32][256];          // staged luma coefficients, 4 KB per warp
    uint8_t luma[kLumaRows][kLumaPitch];          // reconstructed luma tile
    uint8_t c[2][kFTileRows][kCTileCols];         // chroma tile
    TileInfo info;
    uint32_t count[kFusedThreads / 32];
    uint32_t sorted[kFusedThreads];               // blocks by class: DC term | class << 16 | block << 24
};

__device__ __forceinline__ void fill_tile_info(TileInfo& t, const JpegWave& w, uint32_t tile_index) {
    const uint32_t o = owner_of(w.fused_tiles, tile_index);
    const JpegDesc& d = w.descs[w.fused_first + o];
    const uint32_t tile = tile_index - __ldg(w.fused_tiles.first + o);
    const uint32_t tiles_x = (d.width + kColorTileW - 1) / kColorTileW;
    t.ty = tile / tiles_x;
    t.tx = tile - t.ty * tiles_x;
    t.coef = w.coef + (size_t)d.block_off * 64;
    t.info = w.info + d.block_off;
    t.cb = w.planes + d.plane_off[1];
    t.cr = w.planes + d.plane_off[2];
    t.out = w.out + d.out_off;
    t.qq = reinterpret_cast<const uint4*>(w.qt32 + (size_t)d.qt[0] * 32);
    t.mcux = d.mcux; t.mcuy = d.mcuy; t.width = d.width; t.height = d.height; t.cpitch = d.plane_pitch[1];
    t.opitch = d.out_pitch;
}

// Queues the asynchronous copies of the chroma tile: rows cy0-1 .. cy0+8*rows, columns cx0-4 .. cx0+131 as aligned words,
// coordinates clamped to the plane.
__device__ __forceinline__ void queue_chroma_tile(FusedSmem& sm, const TileInfo& t) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int dh = ((int)t.height + 1) / 2;
    const int cx0 = (int)t.tx * (int)(kColorTileW / 2), cy0 = (int)t.ty * 8 * (int)kFusedMcuRows;
    constexpr int kWords = kCTileCols / 4;  // 34
    const int wmax = (int)(t.cpitch / 4) - 1, w0 = cx0 / 4 - 1;
    const int g0 = min(max(w0 + (int)lane, 0), wmax), g1 = min(max(w0 + 32 + (int)lane, 0), wmax);
#pragma unroll
    for (int rr = 0; rr < (kFTileRows + kFusedWarps - 1) / kFusedWarps; ++rr) {
        const int r = (int)warp + kFusedWarps * rr;
        if (r < kFTileRows) {
            const int gy = min(max(cy0 + r - 1, 0), dh - 1);
            const uint32_t* gb = reinterpret_cast<const uint32_t*>(t.cb + (size_t)gy * t.cpitch);
            const uint32_t* gr = reinterpret_cast<const uint32_t*>(t.cr + (size_t)gy * t.cpitch);
            const uint32_t sb = (uint32_t)__cvta_generic_to_shared(&sm.c[0][r][0]);
            const uint32_t sr = (uint32_t)__cvta_generic_to_shared(&sm.c[1][r][0]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sb + lane * 4), "l"(gb + g0) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sr + lane * 4), "l"(gr + g0) : "memory");
            if (lane < kWords - 32) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sb + (32 + lane) * 4), "l"(gb + g1) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sr + (32 + lane) * 4), "l"(gr + g1) : "memory");
            }
        }
    }
}

// The full butterfly needs twice the registers of everything else in the fused kernel and runs for a minority of the
// blocks: it lives in a function of its own, so that it does not set the register count of the whole kernel.
__device__ __noinline__ void idct_full_to_tile(const uint4* rows, uint32_t swz, uint32_t nrows, uint32_t dc, const uint4* qq, uint8_t* dst) {
    uint4 c[8];
    read_block(rows, swz, nrows, dc, c);
    idct_block(c, qq, kClsFull, [&](int r, uint32_t lo, uint32_t hi) {
        *reinterpret_cast<uint2*>(dst + r * kLumaPitch) = make_uint2(lo, hi);
    });
}

#ifndef DG_FUSED_MIN_CTAS
#define DG_FUSED_MIN_CTAS (12 / DG_FUSED_MCU_ROWS)
#endif
__global__ void __launch_bounds__(kFusedThreads, DG_FUSED_MIN_CTAS) k_luma_color(JpegWave w, uint32_t first_tile) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FusedSmem& sm = *reinterpret_cast<FusedSmem*>(smem_raw);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const TileInfo& t = sm.info;  // read where needed: a copy in registers would not fit beside the butterfly

    if (threadIdx.x == 0) fill_tile_info(sm.info, w, first_tile + blockIdx.x);
    let_next_start();
    wait_for_previous();
    __syncthreads();
    // ---- inputs.  Luma coefficients: warp q owns MCU row q / 2 of the tile and MCUs 8 (q % 2) .. + 7 of it, lane l block
    //      l % 4 of MCU l / 4.  MCUs outside the image are replaced by the nearest one inside: their results land in tile
    //      positions no output pixel reads.  Step i copies what the classes cover of the four blocks of MCU i, lane l row
    //      l % 8 of block l / 8 (into the XOR-swizzled layout the IDCT reads back).
    uint32_t v;
    {
        const uint32_t mrow = warp >> 1, half = warp & 1u;
        const uint32_t myc = min(t.ty * kFusedMcuRows + mrow, t.mcuy - 1), mx0 = t.tx * 16 + half * 8;
        const uint32_t mcu_row = myc * t.mcux;
        v = *(t.info + (size_t)(mcu_row + min(mx0 + (lane >> 2), t.mcux - 1)) * 6 + (lane & 3u)) & 0x3FFFFu;
        queue_chroma_tile(sm, t);
        const uint32_t nrows = class_rows((int)(v >> 16));
        const int16_t* row_base = t.coef + (size_t)mcu_row * 384;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bb = i * 4 + (lane >> 3), r = lane & 7;
            const uint32_t mxc = min(mx0 + i, t.mcux - 1);
            if (r < __shfl_sync(0xFFFFFFFFu, nrows, bb)) {
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.coef[warp][bb * 8 + (r ^ (bb & 7))]);
                const void* src = row_base + (size_t)mxc * 384 + lane * 8;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int W = (int)t.width, H = (int)t.height;

    // ---- luma IDCT, one block per thread.  How much of the butterfly a block needs is its class, and a warp runs the path
    //      its least sparse lane needs; so the tile's 256 blocks are sorted by class (counting sort, while the copies are
    //      under way) and thread i then reconstructs the i-th block of that order: all but at most three warps of the CTA
    //      are uniform.
    const uint32_t cls = v >> 16;
    uint32_t ballot_mine;
    {
        const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, cls == 0), b1 = __ballot_sync(0xFFFFFFFFu, cls == 1),
                       b2 = __ballot_sync(0xFFFFFFFFu, cls == 2);
        if (lane == 0) sm.count[warp] = (uint32_t)__popc(b0) | ((uint32_t)__popc(b1) << 10) | ((uint32_t)__popc(b2) << 20);
        ballot_mine = cls == 0 ? b0 : cls == 1 ? b1 : cls == 2 ? b2 : ~(b0 | b1 | b2);
    }
    __syncthreads();  // class counts are in shared memory
    {
        // per-class counts in 10-bit fields (a sum is at most 256; the fourth class is the rest): before this warp, in total
        uint32_t before = 0, total = 0;
#pragma unroll
        for (int i = 0; i < kFusedThreads / 32; ++i) { const uint32_t n = sm.count[i]; if (i < (int)warp) before += n; total += n; }
        const uint32_t t0 = total & 1023u, t1 = (total >> 10) & 1023u, t2 = total >> 20;
        const uint32_t p0 = before & 1023u, p1 = (before >> 10) & 1023u, p2 = before >> 20;
        uint32_t pos = cls == 0 ? p0 : cls == 1 ? t0 + p1 : cls == 2 ? t0 + t1 + p2 : t0 + t1 + t2 + (warp * 32u - p0 - p1 - p2);
        pos += __popc(ballot_mine & ((1u << lane) - 1u));
        sm.sorted[pos & (kFusedThreads - 1)] = v | (uint32_t)threadIdx.x << 24;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // every thread's copies have landed, and the order is there
    chroma_tile_edges(sm.c, (int)t.tx, (W + 1) / 2);
    {
        const uint32_t mine = sm.sorted[threadIdx.x], blk = mine >> 24;
        const int own = (int)((mine >> 16) & 3u), wcls = warp_class(own);
        const uint32_t nrows = class_rows(own);
        // where block blk was staged, and where it lies in the tile (from the lane / warp that staged it)
        const uint32_t bw = blk >> 5, bl = blk & 31u, swz = bl & 7u;
        const uint4* rows = &sm.coef[bw][bl * 8];
        const uint32_t bx = (bw & 1u) * 16 + (bl >> 2) * 2 + (bl & 1u), by = (bw >> 1) * 2 + ((bl >> 1) & 1u);
        uint8_t* dst = &sm.luma[by * 8][bx * 8];
        if (wcls == kClsFull) {
            idct_full_to_tile(rows, swz, nrows, mine, t.qq, dst);
        } else {
            uint4 c[8];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                uint2 q = make_uint2(0, 0);
                if ((uint32_t)r < nrows) q = *reinterpret_cast<const uint2*>(&rows[r ^ swz]);
                c[r].x = q.x; c[r].y = q.y;
            }
            c[0].x = (c[0].x & 0xFFFF0000u) | (mine & 0xFFFFu);
            idct_block(c, t.qq, wcls, [&](int r, uint32_t lo, uint32_t hi) {
                *reinterpret_cast<uint2*>(dst + r * kLumaPitch) = make_uint2(lo, hi);
            });
        }
    }
    __syncthreads();  // the luma tile and the chroma tile's edges are complete

    // ---- upsampling + colour conversion.  Output rows 2j+1 and 2j+2 read the same two chroma rows with the near / far
    //      weights exchanged, so a thread converts such a pair at a time (pair p of the tile = tile rows 2p-1 and 2p,
    //      chroma tile rows p and p+1).  The tile's first row is the second half of pair 0 and its last row the first
    //      half of the pair after the last whole one: warp 0 converts those two halves in an extra step.
    const int x = (int)t.tx * (int)kColorTileW + (int)lane * 8;
    const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, x < W);
    if (x >= W) return;
    const int npx = min(8, W - x);
    const int cl = (int)lane * 4 + 4;
    const int y0 = (int)t.ty * kLumaRows;
    // everything the loop needs from the tile record, once; x * 3 is a multiple of 8, so all rows of a thread are
    // 8-byte aligned when the image and its pitch are
    const uint32_t opitch = t.opitch;
    uint8_t* const obase = t.out + (size_t)x * 3;
    const bool wide = npx == 8 && ((reinterpret_cast<uintptr_t>(obase) | opitch) & 7u) == 0;
    auto store = [&](int y, const uint32_t (&px)[6]) {
        uint8_t* o = obase + (size_t)y * opitch;
        if (wide) {
            uint2* o2 = reinterpret_cast<uint2*>(o);
            __stcs(o2, make_uint2(px[0], px[1])); __stcs(o2 + 1, make_uint2(px[2], px[3])); __stcs(o2 + 2, make_uint2(px[4], px[5]));
        } else {
            store_rgb8(o, px, npx, lanes);
        }
    };
#pragma unroll 1
    for (int m = 0; m <= kLumaRows / 2 / kFusedWarps; ++m) {
        const int p = (int)warp + kFusedWarps * m;
        if (p > kLumaRows / 2) break;
        const int yA = y0 + 2 * p - 1, yB = yA + 1;
        const bool doA = p > 0 && yA < H, doB = p < kLumaRows / 2 && yB < H;
        if (!doA && !doB) break;
        uint32_t a[8], b[8];
        chroma_pair<kFTileRows>(sm.c, p, cl, a, b);
        uint32_t px[6];
        if (doA) {
            const uint2 ya = *reinterpret_cast<const uint2*>(&sm.luma[2 * p - 1][lane * 8]);
            ycc_to_rgb8(ya.x, ya.y, a, px);
            store(yA, px);
        }
        if (doB) {
            const uint2 yb = *reinterpret_cast<const uint2*>(&sm.luma[2 * p][lane * 8]);
            ycc_to_rgb8(yb.x, yb.y, b, px);
            store(yB, px);
        }
    }
}

// One CTA per tile: a persistent loop over tiles with the next tile's inputs prefetched measured slower, because resident
// CTAs then keep the other stream's entropy decoders off the SMs for a whole launch.
void launch_luma_color(const JpegWave& w, uint32_t first_tile, uint32_t count, cudaStream_t s) {
    if (!count) return;
    static std::once_flag done[64];  // per device: the kernel's shared memory exceeds the default limit
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    std::call_once(done[dev], [] { cudaFuncSetAttribute(k_luma_color, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FusedSmem)); });
    launch_after(k_luma_color, count, kFusedThreads, sizeof(FusedSmem), s, w, first_tile);
}

}  // namespace dg
