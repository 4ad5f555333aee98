// Launch interface between the batch scheduler (api.cu) and the sm_100a kernels.
#pragma once
#include <cuda_runtime.h>

#include "desc.h"

namespace dg {

// Maps a flat work index (block, tile, segment) to its owner (image, pass): first[owner] <= idx < first[owner + 1].
// coarse[idx >> shift] is the owner of work item (idx >> shift) << shift, so the search is a short forward walk.
struct OwnerMap {
    const uint32_t* first;   // n + 1 entries
    const uint32_t* coarse;
    uint32_t n, shift, total;
};

constexpr uint32_t kSms = 148;  // of a B200

#ifdef __CUDACC__
// ---- launches that overlap the end of the kernel before them --------------------------------------------------------------
// A batch is a chain of ten or more kernels, many of them shorter than 20 us when the batch is small.  All of them are launched with
// programmatic stream serialisation: a kernel may start while the one before it ends.  Rules:
//   * every thread calls wait_for_previous() before it reads what an earlier kernel wrote, before it writes anything, and before
//     it returns (so the end of a kernel implies the end of all kernels before it);
//   * before that it may read what the host uploaded: descriptors, owner maps, code, quantisation and filter tables;
//   * what earlier kernels wrote is read with plain loads: by dereferencing a pointer, or with load_global(), whose pointer (or the
//     descriptor it comes out of) passes through from_previous() after the wait.  __ldg() is for what the host uploaded and for
//     memory of the caller: it wants memory that nobody writes while the kernel lives, and a kernel lives from before the one
//     before it has ended.
//   * the reconstruction and resize kernels call let_next_start() first when they have few CTAs: the next kernel then fetches its
//     descriptors and weights meanwhile.  Large grids do not: it would only hand over places that other streams can use.  Nor do
//     the entropy kernels, whose successors want much shared memory and sit in it until the slowest stream is through (256 files:
//     3 810 us a pass against 3 571; one photo 314 against 280).
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() {
    if (gridDim.x <= 2 * kSms) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class T> __device__ __forceinline__ T* from_previous(T* p) {
    asm volatile("" : "+l"(p));
    return p;
}
// Plain loads that name the address space, which the compiler does not know of a pointer that it finds in memory: with its generic
// loads a resize whose windows are too long for the tensor cores took 95 us instead of 83 (2 403 x 2 403 gray pixels to 224).
// The compiler may move them like __ldg(), but not ahead of from_previous(): with volatile ones such resizes took 4 % longer.
__device__ __forceinline__ uint32_t load_global(const uint8_t* p) {
    uint32_t v;
    asm("ld.global.u8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t load_global(const uint32_t* p) {
    uint32_t v;
    asm("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 load_global(const uint2* p) {
    uint2 v;
    asm("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 load_global(const uint4* p) {
    uint4 v;
    asm("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
template <class... P, class... A>
void launch_after(void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t at{};
    at.gridDim = dim3(grid); at.blockDim = dim3(block); at.dynamicSmemBytes = smem; at.stream = s;
    at.attrs = &overlap; at.numAttrs = 1;
    cudaLaunchKernelEx(&at, kernel, P(args)...);
}
#endif

// ---- entropy decoding: work splits (see kernels_huff.cu) ------------------------------------------------------------------
constexpr uint32_t kUnstuffTile = 4096;  // bytes of an entropy-coded segment per CTA of the unstuffing kernels
// bits of an unstuffed stream per thread of the value decoder; the short form while all threads are resident at once
constexpr int kCellBits = 1024, kShortCellBits = 512;
// threads per CTA of the value decoders, one per cell or restart segment: the second form once there is more than the chip holds
// of the first at a time.  Shared memory bounds the warps of an SM (128 bytes of block buffer and up to 128 of stream per
// thread, 18 KB of tables per CTA): four CTAs of 128 threads, or three of 224.
constexpr uint32_t kDecodeThreads = 128, kDecodeThreadsMany = 224;
inline uint32_t decode_threads(uint64_t threads) { return threads > kSms * 4ull * kDecodeThreads ? kDecodeThreadsMany : kDecodeThreads; }
// synchronising decoder: threads per CTA, the entries of the candidate array per cell, and the cells of a span once a thread
// per cell and block of the MCU would be more than the chip holds at once
constexpr uint32_t kGuessLanes = 384, kCandidates = 6, kGuessSpan = 4;
constexpr uint64_t kGuessSpanThreads = kSms * 2048ull;
// Threads of the linking kernel per image.  With an image for most SMs or more, 256 leave the most room for other kernels beside
// them (1024 files of 0.4 Mbit: 3.37 ms a pass against 3.48 with 1024 threads; 256 files of 5 Mbit: 4.29 against 4.30); with fewer,
// an image gets 1024, so that its threads' runs are short.
constexpr uint32_t kMixedRun = 4;
inline uint32_t chain_threads(size_t images) { return images >= 120 ? 256 : 1024; }
// spans of cells a CTA takes, each with a thread per block of the MCU: what the threads allow, 256 staged cells at most
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t guess_spans(uint32_t bpm, uint32_t span) {
    const uint32_t lanes = kGuessLanes / bpm, stage = span == 1 ? 128u : 256u / span;
    return lanes < stage ? lanes : stage;
}
constexpr uint32_t kCodeTablesBytes = 20544;  // look-up tables of one (DC, AC) pair of Huffman tables
// Bit positions are 32-bit numbers.  A stream counts up to this length, which leaves room for what the decoders add to a
// position at its end (the cells of a CTA, a block); what lies behind is as good as cut off.
constexpr uint32_t kMaxStream = (1u << 29) - (1u << 16);
constexpr uint32_t kStreamPad = 512;     // bytes behind an image's unstuffed stream that the bit readers may touch

// How much of a block is non-zero decides how much of the inverse DCT is needed: everything, the top-left 4x4 or 2x2
// coefficients, the DC term alone.
enum : int { kClsFull = 0, kCls4x4 = 1, kCls2x2 = 2, kClsDc = 3 };
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t class_rows(int cls) { return cls == kClsFull ? 8u : cls == kCls4x4 ? 4u : cls == kCls2x2 ? 2u : 0u; }  // rows of coef[] it covers

struct JpegWave {
    const JpegDesc* descs;   // device, n images
    uint32_t n;
    const uint8_t* raw;      // compressed blob
    OwnerMap us_tiles;       // kUnstuffTile-byte pieces of the images' entropy-coded segments; owner = image
    uint32_t* tile_info;     // [us_tiles.total] what each tile keeps
    uint8_t* us;             // unstuffed streams, as big-endian 32-bit words
    uint32_t* us_len;        // [n] bytes of each unstuffed stream
    uint32_t* seg_start;     // restart-segment starts (bytes into the image's unstuffed stream)
    uint32_t* seg_found;     // [n] segments actually present
    uint2* cells;            // of a restart-free stream: -, its blocks; then per cell (see CellOrder): bit position of its first
                             // block, index of that block
    uint4* cand;             // [cells][kCandidates / 2], see CellOrder: two candidates: entry state | exit state << 16, blocks that
                             // start in the cell (see k_huff_guess); lies over what is written after the entropy stage
    int16_t* coef;           // [blocks][64], scan order, natural order inside a block; AC terms, rows the class covers
    uint32_t* diff;          // [blocks] restart-free images: DC difference | class << 16
    uint32_t* info;          // [blocks] DC coefficient (low half) | class << 16
    uint8_t* planes;         // component planes after the IDCT
    uint8_t* out;            // decoded images
    uint32_t* status;        // [items of the batch]
    unsigned long long* spec_stats;  // [0] cells, [1] rounds of the linking kernel, [2] decodes of a cell (candidates, open states, values)
    const HuffTable* huff;   // table pool
    const uint2* table_pairs; uint32_t n_pairs;  // the (DC, AC) pairs of tables the images of the wave use
    uint8_t* codes;          // [n_pairs] look-up tables made from them, kCodeTablesBytes each
    uint32_t max_pairs;      // most distinct pairs one image of the wave uses
    const uint32_t* qt32;    // quantisation pool, 32 words per table: word i holds q[2i] in byte 0 and q[2i+1] in byte 3
    // restart-free images of this wave, longest first; CTAs of the synchronising decoder and the value decoder: owner =
    // index into spec_list
    const uint32_t* spec_list; uint32_t n_spec;
    OwnerMap guess_ctas, write_ctas;
    uint32_t cell_bits;      // kCellBits or kShortCellBits
    uint32_t write_cells, restart_segs;  // cells / segments per CTA of the value decoders: kDecodeThreads or kDecodeThreadsMany
    uint32_t guess_span;     // cells a thread of the synchronising decoder goes through
    uint32_t chain_threads;  // of the linking kernel per image, see chain_threads()
    uint32_t mixed;          // see CellOrder: 1024 linking threads, and more than kMixedRun cells for one of them
    // restart-interval images: restart_segs segments per CTA, owner = index into restart_list
    OwnerMap restart_ctas;
    const uint32_t* restart_list;
    OwnerMap blocks;         // owner = image
    OwnerMap color_tiles;    // owner = image
    // Images [fused_first, n) of the wave are three-component 4:2:0 images at least five pixels wide: they take the fused
    // path (chroma-only IDCT into planes, then one kernel for luma IDCT + upsampling + colour conversion) and are not
    // covered by `blocks` / `color_tiles`.  Owner o of these two maps is image fused_first + o.
    uint32_t fused_first;
    OwnerMap fused_chroma;   // flat index over the chroma blocks (Cb, Cr of MCU 0, Cb, Cr of MCU 1, ...)
    OwnerMap fused_tiles;    // colour tiles, color_tiles() per image
};

void launch_unstuff(const JpegWave& w, cudaStream_t s);
void launch_huff_restart(const JpegWave& w, cudaStream_t s);
void launch_huff_guess(const JpegWave& w, cudaStream_t s);
void launch_huff_chain(const JpegWave& w, cudaStream_t s);
void launch_huff_write(const JpegWave& w, cudaStream_t s);  // all restart-free images, once launch_huff_chain has covered them
void launch_whole_blocks(const JpegWave& w, uint32_t nblocks, cudaStream_t s);
// blocks [first, first + count) of the wave / colour tiles [first, first + count): callers may launch them in groups of
// images (the planes written by the IDCT are then still in L2 when the colour kernel reads them) or once per wave
void launch_idct(const JpegWave& w, uint32_t first, uint32_t count, cudaStream_t s);
void launch_color(const JpegWave& w, uint32_t first_tile, uint32_t count, cudaStream_t s);
// the fused path: chroma blocks [first, first + count) of fused_chroma, tiles [first, first + count) of fused_tiles
void launch_idct_chroma(const JpegWave& w, uint32_t first, uint32_t count, cudaStream_t s);
void launch_luma_color(const JpegWave& w, uint32_t first_tile, uint32_t count, cudaStream_t s);
// whether an image takes the fused path
inline bool fused_decode(uint32_t ncomp, uint32_t hs, uint32_t vs, uint32_t width) { return ncomp == 3 && hs == 2 && vs == 2 && width >= 5; }

// The colour kernel gives one CTA 256 pixels of four MCU rows.
constexpr uint32_t kColorTileW = 256, kColorMcuRows = 4;
inline uint32_t color_tiles(uint32_t width, uint32_t mcuy) {
    // one more row of tiles than the MCU rows need: the 4:2:0 path of the colour kernel shifts its tiles up by one pixel
    // row, so that every pair of output rows that shares its two chroma rows falls into one tile
    return ((width + kColorTileW - 1) / kColorTileW) * (mcuy / kColorMcuRows + 1);
}
#ifndef DG_FUSED_MCU_ROWS
#define DG_FUSED_MCU_ROWS 4
#endif
constexpr uint32_t kFusedMcuRows = DG_FUSED_MCU_ROWS;  // MCU rows of a tile of the fused kernel (64 threads per MCU row)
inline uint32_t fused_tiles(uint32_t width, uint32_t mcuy) {  // the fused kernel's tiles are aligned to MCU rows
    return ((width + kColorTileW - 1) / kColorTileW) * ((mcuy + kFusedMcuRows - 1) / kFusedMcuRows);
}

// ---- resize ---------------------------------------------------------------------------------------------------------
constexpr uint32_t kConvTileW = 64, kConvTileH = 16;    // horizontal pass: output pixels x rows per CTA
constexpr uint32_t kVTileBytes = 256, kVTileH = 4;      // vertical pass, plain path: output bytes x rows per CTA
constexpr uint32_t kVFastBytes = 1024, kVFastRows = 32; // vertical pass, vector path: 64 x 16-byte columns, 4 x 8 rows
constexpr uint32_t kVFastMaxWindow = 128;
// horizontal pass on the tensor cores (ConvPass::fast == 2): output bytes per strip x rows per chunk; limits of what a CTA
// can stage -- source bytes under one 8-byte output tile, and under a whole strip
constexpr uint32_t kHMmaStrip = 64, kHMmaChunk = 32, kHMmaMaxBand = 256, kHMmaMaxSpan = 1008;  // span: 63 pieces of 16 bytes = 252 words, inside the 256 elements a tensor-map box may have
// vertical pass on the tensor cores (ConvPass::fast == 2): output rows per CTA x bytes of a row per chunk; limits of what a CTA can
// stage -- source rows under the eight output rows of one warp, and under all rows of the CTA
constexpr uint32_t kVMmaRows = 64, kVMmaChunk = 64, kVMmaMaxBand = 256, kVMmaMaxSpan = 704;
inline uint32_t conv_tiles_x(const ConvPass& p, bool vertical) {
    if (!vertical && p.fast == 2) return (p.out_w * p.channels + kHMmaStrip - 1) / kHMmaStrip;
    if (vertical && p.fast == 2) return (p.out_w * p.channels + p.cta_chunks * kVMmaChunk - 1) / (p.cta_chunks * kVMmaChunk);
    if (!vertical) return (p.out_w + kConvTileW - 1) / kConvTileW;
    const uint32_t row_bytes = p.out_w * p.channels;
    return p.fast ? (row_bytes + kVFastBytes - 1) / kVFastBytes : (row_bytes + kVTileBytes - 1) / kVTileBytes;
}
inline uint32_t conv_tiles(const ConvPass& p, bool vertical) {
    const uint32_t rows = !vertical ? (p.fast == 2 ? p.cta_chunks * kHMmaChunk : kConvTileH) : p.fast == 2 ? kVMmaRows : p.fast ? kVFastRows : kVTileH;
    return conv_tiles_x(p, vertical) * ((p.out_h + rows - 1) / rows);
}
// Cuts the passes of one stage into CTA tiles.  A CTA of a tensor-core pass first gathers its weights and then walks
// chunks: two CTAs per resident place of the chip keep its SMs evenly busy to the end, one per place is better where that
// leaves a CTA only a few chunks, and two chunks are the least a CTA gets.  (One image of 1.5 Mpixel: horizontal pass 20.6 us
// at four CTAs per place, 15.7 at two, 10.9 at one; 48 images of 5 Mpixel: 275, 253, 252 us, and 268 with CTAs of 2048 rows.)
#ifndef DG_HMMA_CTAS
#define DG_HMMA_CTAS 3
#endif
constexpr uint32_t kHMmaCtasPerSm = DG_HMMA_CTAS, kVMmaCtasPerSm = 2;
constexpr uint32_t kMmaMinChunks = 2, kMmaFewChunks = 4, kMmaMaxChunks = 64;
inline void cut_pass_tiles(ConvPass* passes, size_t n, bool vertical) {
    uint64_t work = 0;  // chunks of all CTAs together
    auto rows_of_ctas = [&](const ConvPass& p) -> uint64_t { return vertical ? (p.out_h + kVMmaRows - 1) / kVMmaRows : (p.out_w * p.channels + kHMmaStrip - 1) / kHMmaStrip; };
    auto chunks_of = [&](const ConvPass& p) -> uint64_t { return vertical ? (p.out_w * p.channels + kVMmaChunk - 1) / kVMmaChunk : (p.out_h + kHMmaChunk - 1) / kHMmaChunk; };
    for (size_t i = 0; i < n; ++i)
        if (passes[i].fast == 2) work += rows_of_ctas(passes[i]) * chunks_of(passes[i]);
    const uint64_t places = kSms * (vertical ? kVMmaCtasPerSm : kHMmaCtasPerSm), one = (work + places - 1) / places;
    uint64_t chunks = (one + 1) / 2;
    if (chunks < kMmaFewChunks) chunks = one < kMmaFewChunks ? one : kMmaFewChunks;
    chunks = chunks < kMmaMinChunks ? kMmaMinChunks : chunks > kMmaMaxChunks ? kMmaMaxChunks : chunks;
    for (size_t i = 0; i < n; ++i) {
        ConvPass& p = passes[i];
        if (p.fast == 2) {  // as few CTAs as that gives, as equal as they get
            const uint64_t all = chunks_of(p), ctas = (all + chunks - 1) / chunks;
            p.cta_chunks = (uint32_t)((all + ctas - 1) / ctas);
        }
        p.tiles_x = conv_tiles_x(p, vertical);
    }
}
constexpr uint32_t kCopyTileBytes = 4096;
inline uint32_t copy_tiles(const CopyJob& j) {  // tiles start at multiples of 16 of the destination's address
    return (uint32_t)(((uint64_t)j.row_bytes * j.rows + 15 + kCopyTileBytes - 1) / kCopyTileBytes);
}

// the passes that take the tensor-core kernel (fast == 2) come first in `passes` and own tiles [0, mma_tiles).  timeouts: counts
// the CTAs of those kernels that ran out of patience waiting for a copy (never expected; it exists so that a wait can be
// bounded without the failure going unnoticed).
void launch_conv_h(const ConvPass* passes, OwnerMap map, const uint32_t* tables, uint32_t mma_tiles, unsigned int* timeouts, cudaStream_t s);
void launch_conv_v(const ConvPass* passes, OwnerMap map, const uint32_t* tables, uint32_t mma_tiles, unsigned int* timeouts, cudaStream_t s);
void launch_copy(const CopyJob* jobs, OwnerMap map, cudaStream_t s);
constexpr uint32_t kAlphaTilePx = 2048;  // pixels per CTA of the alpha multiply / divide kernel
void launch_alpha(const AlphaJob* jobs, OwnerMap map, cudaStream_t s);
constexpr uint32_t kToRgbTilePx = 2048;  // pixels per CTA of the RGB8 conversion
void launch_to_rgb8(const ToRgbJob* jobs, OwnerMap map, cudaStream_t s);

}  // namespace dg
