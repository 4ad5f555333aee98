// Baseline JPEG entropy decoding on sm_100a: byte unstuffing, Huffman decode, DC prediction.  First half of the decode
// datago reaches through image::load_from_memory (src/worker_wds.rs:45) / ImageReader::decode (src/worker_files.rs:14-16).
//
// Output of this file, per 8x8 block in scan (MCU-interleaved) order:
//   info[block]  low half: the DC coefficient (int16, prediction resolved); bits 16-17: the block's class
//   coef[block]  64 int16 in natural order, DC slot zero -- only the rows the class covers are written (and read)
// The class says where the AC coefficients end (kClsFull / kCls4x4 / kCls2x2 / kClsDc).  On photographs at ordinary
// qualities half of the blocks or more carry a handful of low-frequency coefficients or none, so keeping the DC terms
// dense and skipping the rows that hold nothing is worth several times the memory traffic of whole blocks, and nothing has
// to be zeroed before or after.
#include <cooperative_groups.h>

#include <cstdint>
#include <mutex>

#include "kernels.h"

namespace cg = cooperative_groups;

namespace dg {

namespace {

__device__ const uint8_t kNatural[64] = {0,  1,  8,  16, 9,  2,  3,  10, 17, 24, 32, 25, 18, 11, 4,  5,
                                         12, 19, 26, 33, 40, 48, 41, 34, 27, 20, 13, 6,  7,  14, 21, 28,
                                         35, 42, 49, 56, 57, 50, 43, 36, 29, 22, 15, 23, 30, 37, 44, 51,
                                         58, 59, 52, 45, 38, 31, 39, 46, 53, 60, 61, 54, 47, 55, 62, 63};

__device__ __forceinline__ uint32_t owner_of(const OwnerMap& m, uint32_t idx) {
    uint32_t o = __ldg(m.coarse + (idx >> m.shift));
    while (o + 1 < m.n && __ldg(m.first + o + 1) <= idx) ++o;
    return o;
}

__device__ __forceinline__ uint32_t shr_clamp(uint32_t x, uint32_t n) {  // shift counts >= 32 give 0
    uint32_t r;
    asm("shr.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}
// shared-memory reads by 32-bit address (volatile: the memory behind them changes under asynchronous copies)
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

}  // namespace

// ---------------------------------------------------------------------------------------------------------------
// K0  unstuff: drops stuffed zeros (FF 00 -> FF), fill bytes and RSTn markers from the entropy-coded segments, records
//     where each restart segment starts in the compacted stream and stops at the first other marker (EOI).  The
//     compacted stream is stored as big-endian 32-bit words, the form the bit readers want.
//     One CTA per 4 KB tile of an image, in two launches: the first counts what each tile keeps, the second adds up the
//     counts of the tiles before its own (a few hundred words at most for ordinary files) and writes.  One CTA walking a
//     whole file step by step, as before, lasted as long as the longest file (1.25 ms for 2.2 MB).
// ---------------------------------------------------------------------------------------------------------------
constexpr int kUnstuffThreads = 256;

namespace {

// tile_info: bits 0-12 bytes kept, 13-25 restart markers, 26 the scan ends in this tile
constexpr uint32_t kTileRstShift = 13, kTileTerm = 1u << 26, kTileMask = 0x1FFFu;

// four flags, one per byte of m (0xFF or 0x00 each), as bits 0..3
__device__ __forceinline__ uint32_t byte_flags(uint32_t m) { return __dp4a(m & 0x08040201u, 0x01010101u, 0u); }

// The calling thread's 16 bytes at i0 classified: which are kept, which begin a restart marker, and whether (where) the
// scan ends among them.  next / prev: the bytes around them.
struct Unit { uint32_t w[4]; uint32_t keep, rst, term; };
__device__ __forceinline__ Unit classify(const uint8_t* in, uint32_t i0, uint32_t len) {
    Unit u;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (i0 < len) v = __ldg(reinterpret_cast<const uint4*>(in + i0));  // blob slices are padded to 16 bytes with zeros
    u.w[0] = v.x; u.w[1] = v.y; u.w[2] = v.z; u.w[3] = v.w;
    const uint32_t prev = (i0 > 0 && i0 <= len) ? __ldg(in + i0 - 1) : 0u;
    const uint32_t next = (i0 + 16 < len) ? __ldg(in + i0 + 16) : 0u;
    uint32_t F = 0, Z = 0, R = 0;  // FF bytes, zero bytes, bytes D0..D7
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        F |= byte_flags(__vcmpeq4(u.w[k], 0xFFFFFFFFu)) << (4 * k);
        Z |= byte_flags(__vcmpeq4(u.w[k], 0u)) << (4 * k);
        R |= byte_flags(__vcmpeq4(u.w[k] & 0xF8F8F8F8u, 0xD0D0D0D0u)) << (4 * k);
    }
    const uint32_t valid = i0 >= len ? 0u : len - i0 >= 16 ? 0xFFFFu : (1u << (len - i0)) - 1u;
    const uint32_t nF = (F >> 1) | (next == 0xFFu ? 0x8000u : 0u), nZ = (Z >> 1) | (next == 0u ? 0x8000u : 0u),
                   nR = (R >> 1) | ((next & 0xF8u) == 0xD0u ? 0x8000u : 0u);
    const uint32_t pF = (F << 1) | (prev == 0xFFu ? 1u : 0u);
    u.keep = ((F & nZ) | (~F & ~(pF & (Z | R)))) & valid;
    u.rst = F & nR & ~nZ & valid;
    u.term = F & ~nZ & ~nF & ~nR & valid;
    return u;
}

}  // namespace

__global__ void __launch_bounds__(kUnstuffThreads) k_unstuff_count(JpegWave w) {
    const uint32_t o = owner_of(w.us_tiles, blockIdx.x);
    const JpegDesc& d = w.descs[o];
    const uint32_t tile = blockIdx.x - __ldg(w.us_tiles.first + o);
    __shared__ uint32_t s_end, s_sum;
    if (threadIdx.x == 0) { s_end = 0xFFFFFFFFu; s_sum = 0; }
    const uint32_t i0 = tile * kUnstuffTile + threadIdx.x * 16;
    Unit u = classify(w.raw + d.raw_off, i0, d.raw_len);
    if (__syncthreads_or(u.term != 0)) {  // nothing at or after the terminating marker survives
        if (u.term) atomicMin(&s_end, i0 + __ffs(u.term) - 1);
        __syncthreads();
        const uint32_t end = s_end, m = end <= i0 ? 0u : end - i0 >= 16 ? 0xFFFFu : (1u << (end - i0)) - 1u;
        u.keep &= m; u.rst &= m;
    }
    const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popc(u.keep) | ((uint32_t)__popc(u.rst) << kTileRstShift));
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, sum);
    __syncthreads();
    if (threadIdx.x == 0) w.tile_info[blockIdx.x] = s_sum | (s_end != 0xFFFFFFFFu ? kTileTerm : 0u);
}

__global__ void __launch_bounds__(kUnstuffThreads) k_unstuff_write(JpegWave w) {
    const uint32_t o = owner_of(w.us_tiles, blockIdx.x);
    const JpegDesc& d = w.descs[o];
    const uint32_t tile0 = __ldg(w.us_tiles.first + o), ntile = __ldg(w.us_tiles.first + o + 1) - tile0, tile = blockIdx.x - tile0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t* const out = w.us + d.us_off;
    uint32_t* const seg = w.seg_start + d.seg_off;
    __shared__ uint32_t s_end, s_term, s_kept, s_rst;
    __shared__ uint32_t s_warp[kUnstuffThreads / 32];
    __shared__ __align__(16) uint8_t s_out[kUnstuffTile + 32];
    if (tid == 0) { s_end = 0xFFFFFFFFu; s_term = 0xFFFFFFFFu; s_kept = 0; s_rst = 0; }
    __syncthreads();
    const uint32_t i0 = tile * kUnstuffTile + tid * 16;
    Unit u = classify(w.raw + d.raw_off, i0, d.raw_len);
    // what the tiles before this one kept
    uint32_t kept = 0, rst = 0;
    bool ended = false;
    for (uint32_t t = tid; t < tile; t += kUnstuffThreads) {
        const uint32_t v = w.tile_info[tile0 + t];
        kept += v & kTileMask; rst += (v >> kTileRstShift) & kTileMask;
        if (v & kTileTerm) { ended = true; atomicMin(&s_term, t); }
    }
    if (u.term) atomicMin(&s_end, i0 + __ffs(u.term) - 1);
    ended = __syncthreads_or(ended);
    if (ended) {  // data behind the end of the scan: only the tiles up to the terminating one count
        kept = rst = 0;
        for (uint32_t t = tid; t <= s_term; t += kUnstuffThreads) {
            const uint32_t v = w.tile_info[tile0 + t];
            kept += v & kTileMask; rst += (v >> kTileRstShift) & kTileMask;
        }
        u.keep = u.rst = 0;
    } else if (s_end != 0xFFFFFFFFu) {
        const uint32_t end = s_end, m = end <= i0 ? 0u : end - i0 >= 16 ? 0xFFFFu : (1u << (end - i0)) - 1u;
        u.keep &= m; u.rst &= m;
    }
    if (tile > 0) {
        kept = __reduce_add_sync(0xFFFFFFFFu, kept);
        rst = __reduce_add_sync(0xFFFFFFFFu, rst);
        if (lane == 0 && (kept | rst)) { atomicAdd(&s_kept, kept); atomicAdd(&s_rst, rst); }
    }
    // exclusive scan of (restart count << 16 | kept count) over the CTA
    const uint32_t mine = ((uint32_t)__popc(u.rst) << 16) | (uint32_t)__popc(u.keep);
    uint32_t inc = mine;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, k); if (lane >= k) inc += t; }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    const uint32_t base = s_kept, rbase = s_rst;
    uint32_t wpre = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < kUnstuffThreads / 32; ++i) { const uint32_t t = s_warp[i]; if (i < warp) wpre += t; tot += t; }
    const uint32_t excl = wpre + inc - mine, n = tot & 0xFFFFu;
    // the tile's bytes in shared memory at the alignment they have in the stream (stream byte b at s_out[b - aligned base])
    const uint32_t lead = base & 15u;
    uint32_t pos = lead + (excl & 0xFFFFu);
    if (u.keep == 0xFFFFu) {
#pragma unroll
        for (int j = 0; j < 16; ++j) s_out[(pos + j) ^ 3u] = (uint8_t)(u.w[j >> 2] >> (8 * (j & 3)));
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if ((u.keep >> j) & 1u) { s_out[pos ^ 3u] = (uint8_t)(u.w[j >> 2] >> (8 * (j & 3))); ++pos; }
        if (u.rst) {
            uint32_t r = rbase + (excl >> 16);
            for (uint32_t m = u.rst; m; m &= m - 1) {
                const uint32_t before = m & (0u - m);
                ++r;
                if (r < d.nseg) seg[r] = base + (excl & 0xFFFFu) + __popc(u.keep & (before - 1));
            }
        }
    }
    __syncthreads();
    uint8_t* const ob = out + (base - lead);
    const uint32_t end = lead + n;  // s_out holds bytes [lead, end)
    for (uint32_t q = tid; q * 16 < end; q += kUnstuffThreads) {
        if (q * 16 >= lead && q * 16 + 16 <= end) reinterpret_cast<uint4*>(ob)[q] = reinterpret_cast<const uint4*>(s_out)[q];
        else  // a piece shared with a neighbouring tile: byte by byte
            for (uint32_t k = max(q * 16, lead); k < min(q * 16 + 16, end); ++k) ob[k ^ 3u] = s_out[k ^ 3u];
    }
    if (tile == 0 && tid == 0) seg[0] = 0;
    if (tile + 1 == ntile) {
        const uint32_t total = base + n;
        if (tid < 32) out[(total + tid) ^ 3u] = 0;  // the bit readers may look a few bytes past the end
        if (tid == 0) { w.us_len[o] = total; w.seg_found[o] = rbase + (tot >> 16) + 1; }
    }
}

void launch_unstuff(const JpegWave& w, cudaStream_t s) {
    if (!w.n) return;
    k_unstuff_count<<<w.us_tiles.total, kUnstuffThreads, 0, s>>>(w);
    k_unstuff_write<<<w.us_tiles.total, kUnstuffThreads, 0, s>>>(w);
}

// ---------------------------------------------------------------------------------------------------------------
// K1  Huffman entropy decode of images without restart markers, in two kernels.
//
// The only decoder state between two blocks is (bit position p, block index c inside the MCU): the tables and the meaning
// of the next symbol follow from it.  The stream is cut into cells of kCellBits (1024) bits; what the second kernel needs
// is, for every cell, the state at the first block that starts in it and that block's index in the image.
//
//  k_huff_sync   finds those states.  Every thread owns a run of consecutive cells and decodes it from a guessed state
//     (first AC symbol of a luma block at the run's first bit), noting the state at the first block start of each cell
//     and of the next thread's run.  Huffman streams re-synchronise, so the state a thread hands over is usually right
//     even though it started from a guess; each thread then compares what its left neighbour hands over with what it
//     assumed, decodes again from the corrected state where they differ -- only until it meets the recorded state of
//     a cell -- and this repeats until nothing changes (bounded: thread j is final after round j).  Nothing but code
//     lengths matters here, so symbols are looked up two at a time where they fit the table index and no value is ever
//     extracted.  Measured on 4:2:0 photographs the distance to synchronisation is 200 to 800 bits in the median and 3000
//     to 5000 at the 99th percentile (the phase inside the MCU is what takes long: with the 4:4:4 pattern it is 70 and
//     330), so runs of several cells lose little to the second decode; a short image gets short runs instead, because
//     then the latency of one thread's run is what counts.
//     One CTA, or one cluster of CTAs sharing the hand-over states through distributed shared memory, per image.
//  k_huff_write  one thread per cell decodes the blocks that start in it, values included, collects a block in shared
//     memory and writes it out whole: DC difference and class to diff[], the rows the class covers to coef[].
// ---------------------------------------------------------------------------------------------------------------
namespace {

constexpr int kPairBits = 10;       // table index of the symbol-pair look-up
constexpr uint32_t kNoState = 0xFFFFFFFFu;  // "the stream has ended" in place of a bit position

// What follows the fast table: codes longer than it (see HuffTable::limit).
struct LongCodes {
    uint32_t limit[8];
    int32_t valoff[20];  // 17 used
    uint8_t vals[256];
};
__device__ __forceinline__ void load_long_codes(LongCodes& t, const HuffTable* src, int tid, int nthreads) {
    for (int i = tid; i < 8; i += nthreads) t.limit[i] = __ldg(src->limit + i);
    for (int i = tid; i < 17; i += nthreads) t.valoff[i] = __ldg(src->valoff + i);
    for (int i = tid; i < 64; i += nthreads) reinterpret_cast<uint32_t*>(t.vals)[i] = __ldg(reinterpret_cast<const uint32_t*>(src->vals) + i);
}
// No search: the code length follows from six comparisons against the table's left-aligned limits, the symbol from the
// canonical offset of that length.  Returns length | symbol << 8; 16 with bit 31 set when no code matches.
__device__ __forceinline__ uint32_t long_code(const LongCodes* t, uint32_t top) {
    const uint32_t v = top >> 16;
    const uint4 la = *reinterpret_cast<const uint4*>(&t->limit[0]);
    const uint4 lb = *reinterpret_cast<const uint4*>(&t->limit[4]);
    const uint32_t len = 10u + (v >= la.x) + (v >= la.y) + (v >= la.z) + (v >= la.w) + (v >= lb.x) + (v >= lb.y);
    if (v >= lb.z) return 16u | 0x80000000u;
    return len | ((uint32_t)t->vals[(int32_t)(v >> (16u - len)) + t->valoff[len]] << 8);
}

// The image's tables, each distinct one once: slot of the DC / AC table of component i.
struct TableSlots {
    uint32_t id[6], n;
    uint8_t dc[3], ac[3];
};
__device__ __forceinline__ TableSlots table_slots(const JpegDesc& d) {
    TableSlots t;
    t.n = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int same = -1;
#pragma unroll
        for (int j = 0; j < k; ++j) if (same < 0 && d.dc_tab[j] == d.dc_tab[k]) same = j;
        if (same >= 0) t.dc[k] = t.dc[same]; else { t.dc[k] = (uint8_t)t.n; t.id[t.n++] = d.dc_tab[k]; }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int same = -1;
#pragma unroll
        for (int j = 0; j < k; ++j) if (same < 0 && d.ac_tab[j] == d.ac_tab[k]) same = j;
        if (same >= 0) t.ac[k] = t.ac[same]; else { t.ac[k] = (uint8_t)t.n; t.id[t.n++] = d.ac_tab[k] | 0x80000000u; }
    }
    return t;
}

// One table of the synchronising decoder: index = next kPairBits bits.  Low half: the first symbol alone, high half: the
// first two when the second one's code lies inside the index (else the first again).  A half is bits consumed | slots
// advanced << 5; 64 slots or more end the block.  0: the first code is longer than the fast table.
struct SyncTab {
    uint32_t pair[1 << kPairBits];
    LongCodes lc;
};
static_assert(sizeof(SyncTab) % 16 == 0, "tables follow one another in shared memory");

constexpr int kRingPitch = 144;  // bytes per thread: eight 16-byte pieces of its stream, padded against bank conflicts

template <int T>
struct SyncMisc {
    uint2 exit[T];         // state each thread hands to its right neighbour
    uint32_t tabs[8];      // per block of the MCU: byte offset of its DC table | AC table << 16
    uint32_t warp[32];
    uint32_t flag[3];      // cluster: some thread still differs (by round, modulo 3)
    uint32_t total;        // blocks found by this CTA's threads
};

}  // namespace

template <int T, bool CLUSTER>
__global__ void __launch_bounds__(T) k_huff_sync(JpegWave w, uint32_t first) {
    extern __shared__ __align__(16) unsigned char sync_smem[];
    unsigned char* const ring0 = sync_smem;
    SyncMisc<T>& sh = *reinterpret_cast<SyncMisc<T>*>(sync_smem + T * kRingPitch);
    unsigned char* const tab0 = sync_smem + T * kRingPitch + sizeof(SyncMisc<T>);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t rank = 0, nrank = 1;
    if (CLUSTER) { rank = cg::this_cluster().block_rank(); nrank = cg::this_cluster().num_blocks(); }
    const uint32_t img = w.spec_list[first + blockIdx.x / nrank];
    const JpegDesc& d = w.descs[img];

    const uint32_t bpm = d.bpm;
    {
        const TableSlots ts = table_slots(d);
        for (uint32_t t = 0; t < ts.n; ++t) {
            const HuffTable* src = w.huff + (ts.id[t] & 0x7FFFFFFFu);
            const bool is_ac = (ts.id[t] >> 31) != 0;
            SyncTab& dst = *reinterpret_cast<SyncTab*>(tab0 + t * sizeof(SyncTab));
            for (uint32_t i = tid; i < (1u << kPairBits); i += T) {
                const uint32_t e1 = __ldg(src->lut + (i >> (kPairBits - kLutBits)));
                uint32_t one = 0, two = 0;
                if (e1) {
                    const uint32_t u1 = e1 & 63u, s1 = (e1 >> 11) & 15u, r1 = (e1 >> 15) & 15u;
                    const uint32_t a1 = !is_ac ? 1u : (s1 || r1 == 15u) ? r1 + 1u : 64u;
                    one = two = u1 | a1 << 5;
                    if (is_ac && a1 < 64u && u1 < (uint32_t)kPairBits) {
                        const uint32_t e2 = __ldg(src->lut + (((i << u1) & ((1u << kPairBits) - 1u)) >> (kPairBits - kLutBits)));
                        if (e2 && ((e2 >> 6) & 31u) <= kPairBits - u1) {
                            const uint32_t s2 = (e2 >> 11) & 15u, r2 = (e2 >> 15) & 15u;
                            two = (u1 + (e2 & 63u)) | (a1 + ((s2 || r2 == 15u) ? r2 + 1u : 64u)) << 5;
                        }
                    }
                }
                dst.pair[i] = one | two << 16;
            }
            load_long_codes(dst.lc, src, tid, T);
        }
        if ((uint32_t)tid < bpm) {
            const uint32_t luma = d.hs * d.vs, comp = (uint32_t)tid < luma ? 0u : tid - luma + 1u;
            sh.tabs[tid] = (uint32_t)(ts.dc[comp] * sizeof(SyncTab)) | (uint32_t)(ts.ac[comp] * sizeof(SyncTab)) << 16;
        }
        if (tid < 3) sh.flag[tid] = 0;
    }
    __syncthreads();

    const uint32_t total = w.us_len[img] * 8u;
    const uint32_t ncell = (total + kCellBits - 1) / kCellBits;
    const uint8_t* const us = w.us + d.us_off;
    uint2* const recs = w.cells + d.cell_off;
    const uint32_t gt = rank * T + tid, nthread = nrank * T;
    const uint32_t run = (ncell + nthread - 1) / nthread;
    const uint32_t kbeg = min(gt * run, ncell), kend = min(kbeg + run, ncell);
    const bool active = kbeg < kend;
    const uint32_t ring = smem_addr(ring0) + tid * kRingPitch, tabs = smem_addr(sh.tabs), tbase = smem_addr(tab0);

    uint32_t found = 0;                       // blocks that start in this thread's cells
    uint2 entry = make_uint2(0, 0), exit = make_uint2(kNoState, 0);

    // Decodes from (p, z, c) to the first block start at or behind the end of the run.  Redoing (REDO), it stops as soon as
    // it meets the state recorded for one of the cells.
    auto decode = [&](uint32_t p, uint32_t z, uint32_t c, bool redo) {
        uint32_t k = kbeg, bound = kbeg * kCellBits;  // the next cell to enter, and where it begins
        uint32_t nb = 0, old_n = 0;                   // blocks since the open cell's entry; what the cell counted before
        bool open = false;
        uint2 at = make_uint2(0, 0);                  // entry state of the open cell
        // a block start at p >= bound, or behind the end of the stream: true when the run is done
        auto enter = [&]() -> bool {
            if (p > total) {  // the block that ended here is not whole
                if (p != kNoState && nb) --nb;
                p = kNoState; c = 0;
            }
            while (p >= bound) {
                uint32_t had_n = 0;
                bool met = false;
                if (k < kend && redo) {
                    const uint2 had = recs[k];
                    had_n = had.y & 0x0FFFFFFFu;
                    met = open && had.x == p && (had.y >> 28) == c;
                }
                if (open) { recs[k - 1] = make_uint2(at.x, at.y << 28 | nb); found += nb - old_n; }
                if (met) return true;
                if (k == kend) { exit = make_uint2(p, c); return true; }
                if (k == kbeg) entry = make_uint2(p, c);
                nb = 0; old_n = had_n; at = make_uint2(p, c); open = true;
                ++k; bound += kCellBits;
            }
            return false;
        };
        if (z == 0 && enter()) return;
        // the stream in pieces of 16 bytes through this thread's ring; a window of three words in registers
        uint32_t wr = p >> 7, wi = p >> 5;
#pragma unroll
        for (int i = 0; i < 8; ++i, ++wr) copy16(ring + (wr & 7u) * 16, us + (size_t)wr * 16);
        copy_commit();
        copy_wait<0>();
        auto word = [&](uint32_t i) { return lds32(ring + ((i << 2) & 124u)); };
        uint32_t w0 = word(wi), w1 = word(wi + 1), w2 = word(wi + 2);
        uint32_t tb = lds32(tabs + c * 4);
        uint32_t tab = tbase + (z ? tb >> 16 : tb & 0xFFFFu);
        for (;;) {
            // A step consumes at most 31 bits, so four of them cross at most one piece and one copy per turn keeps the
            // ring full.  The copies of the last four turns may still be under way: they are at least three pieces ahead.
            if (wr < (p >> 7) + 8) { copy16(ring + (wr & 7u) * 16, us + (size_t)wr * 16); ++wr; }
            copy_commit();
            copy_wait<4>();
#pragma unroll
            for (int step = 0; step < 4; ++step) {
                const uint32_t top = __funnelshift_l(w1, w0, p);
                uint32_t e = lds32(tab + ((top >> (32 - kPairBits)) << 2));
                if (e == 0) {
                    const uint32_t lc = long_code(reinterpret_cast<const LongCodes*>(__cvta_shared_to_generic(tab + (sizeof(uint32_t) << kPairBits))), top);
                    const uint32_t s = (lc >> 8) & 15u, r = (lc >> 12) & 15u;
                    const uint32_t adv = z == 0 ? 1u : (s || r == 15u) ? r + 1u : 64u;
                    e = ((lc & 31u) + s) | adv << 5;
                    e |= e << 16;
                }
                // the second symbol belongs to this block only if the first one does not end it
                const uint32_t h = z + ((e >> 5) & 127u) >= 64u ? e & 0xFFFFu : e >> 16;
                p += h & 31u;
                z += h >> 5;
                tab = tbase + (tb >> 16);
                if (z >= 64u) {
                    z = 0;
                    c = c + 1 == bpm ? 0u : c + 1;
                    tb = lds32(tabs + c * 4);
                    tab = tbase + (tb & 0xFFFFu);
                    ++nb;
                    if (p >= bound || p > total) { if (enter()) return; }
                }
                const uint32_t nwi = p >> 5;
                if (nwi != wi) { w0 = w1; w1 = w2; w2 = word(nwi + 2); wi = nwi; }
            }
        }
    };

    if (active) decode(gt ? kbeg * kCellBits : 0u, gt ? 1u : 0u, 0u, false);
    sh.exit[tid] = exit;
    uint32_t decodes = active ? 1u : 0u, rounds = 1;
    if (CLUSTER) cg::this_cluster().sync(); else __syncthreads();
    const uint32_t limit = nthread + 1;
    uint32_t round = 0;
    for (; round <= limit; ++round) {
        uint2 prev = entry;
        if (active && gt) prev = tid ? sh.exit[tid - 1] : *cg::this_cluster().map_shared_rank(&sh.exit[T - 1], rank - 1);
        const bool need = active && (prev.x != entry.x || prev.y != entry.y);
        bool any = __syncthreads_or(need);
        if (CLUSTER) {
            if (any && tid == 0) *cg::this_cluster().map_shared_rank(&sh.flag[round % 3], 0) = 1;
            cg::this_cluster().sync();
            any = *cg::this_cluster().map_shared_rank(&sh.flag[round % 3], 0) != 0;
            if (rank == 0 && tid == 0) sh.flag[(round + 2) % 3] = 0;
        }
        if (!any) break;
        if (need) {
            ++decodes;
            decode(prev.x, 0, prev.y, true);
            sh.exit[tid] = exit;
        }
        ++rounds;
        if (CLUSTER) cg::this_cluster().sync(); else __syncthreads();
    }
    // index of the first block of every cell
    uint32_t inc = found;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o); if (lane >= o) inc += t; }
    if (lane == 31) sh.warp[warp] = inc;
    decodes = __reduce_add_sync(0xFFFFFFFFu, decodes);
    if (lane == 0) atomicAdd(w.spec_stats + 2, (unsigned long long)decodes);
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int i = 0; i < T / 32; ++i) { const uint32_t v = sh.warp[i]; if (i < warp) before += v; all += v; }
    if (CLUSTER) {
        if (tid == 0) sh.total = all;
        cg::this_cluster().sync();
        for (uint32_t r = 0; r < rank; ++r) before += *cg::this_cluster().map_shared_rank(&sh.total, r);
        cg::this_cluster().sync();  // nobody's shared memory goes away while it is being read
    }
    uint32_t base = before + inc - found;
    for (uint32_t k = kbeg; k < kend; ++k) { const uint32_t n = recs[k].y & 0x0FFFFFFFu; recs[k].y = base; base += n; }
    if (rank + 1 == nrank && tid == T - 1) {
        recs[ncell] = make_uint2(kNoState, base);
        uint32_t err = 0;
        if (base < d.nblocks) err |= kStTruncated;
        if (round > limit) err |= kStSyncLimit;
        if (err) atomicOr(w.status + d.item, err);
        atomicAdd(w.spec_stats, (unsigned long long)max(1u, (ncell + 255u) / 256u));
        atomicAdd(w.spec_stats + 1, (unsigned long long)rounds);
    }
}

// ---- blocks with their values --------------------------------------------------------------------------------------
namespace {

// One table of the value decoder: HuffTable::lut as it is, and the codes beyond it.
struct ValueTab {
    uint32_t lut[1 << kLutBits];
    LongCodes lc;
};
static_assert(sizeof(ValueTab) % 16 == 0, "tables follow one another in shared memory");

constexpr uint32_t kNotDc = 1u << 28, kNot2x2 = 1u << 29, kNot4x4 = 1u << 30;

// Zig-zag position -> byte offset of the coefficient in a lane's block buffer (row r of the lane's block sits at
// r * T * 16: rows of neighbouring lanes are neighbours, so whole-row accesses are conflict free) | class flags.
template <int T>
__device__ __forceinline__ uint32_t place_of(uint32_t zz) {
    const uint32_t nat = kNatural[zz], r = nat >> 3, c = nat & 7u;
    return r * (T * 16) + c * 2 | kNotDc | (r > 1 || c > 1 ? kNot2x2 : 0u) | (r > 3 || c > 3 ? kNot4x4 : 0u);
}

template <int T>
struct ValueMisc {
    uint4 block[8 * T];    // the lanes' current blocks
    uint32_t place[64];
    uint32_t tabs[8];      // per block of the MCU: byte offset of its DC table | AC table << 16
};

// Shared memory of the value decoder: [ValueMisc | tables]; returns the base address of the tables.
template <int T>
__device__ __forceinline__ void value_setup(const JpegWave& w, const JpegDesc& d, ValueMisc<T>& sh, unsigned char* tab0) {
    const int tid = threadIdx.x;
    const TableSlots ts = table_slots(d);
    for (uint32_t t = 0; t < ts.n; ++t) {
        const HuffTable* src = w.huff + (ts.id[t] & 0x7FFFFFFFu);
        ValueTab& dst = *reinterpret_cast<ValueTab*>(tab0 + t * sizeof(ValueTab));
        for (int i = tid; i < (1 << kLutBits) / 4; i += T) reinterpret_cast<uint4*>(dst.lut)[i] = __ldg(reinterpret_cast<const uint4*>(src->lut) + i);
        load_long_codes(dst.lc, src, tid, T);
    }
    if ((uint32_t)tid < d.bpm) {
        const uint32_t luma = d.hs * d.vs, comp = (uint32_t)tid < luma ? 0u : tid - luma + 1u;
        sh.tabs[tid] = (uint32_t)(ts.dc[comp] * sizeof(ValueTab)) | (uint32_t)(ts.ac[comp] * sizeof(ValueTab)) << 16;
    }
    if (tid < 64) sh.place[tid] = place_of<T>(tid);
#pragma unroll
    for (int r = 0; r < 8; ++r) sh.block[r * T + tid] = make_uint4(0, 0, 0, 0);
}

// Decodes blocks [blk, end) of an image from bit p on.  word(i): the i-th big-endian word of the image's stream.
// limit: blocks that reach beyond this bit are not whole -- decoding stops there.  ABSOLUTE: the DC predictors start at
// zero here (a restart segment) and info[] receives the DC terms themselves instead of their differences.
// Returns the blocks decoded.  One code path for DC and AC symbols: the lanes of a warp are at unrelated places.
template <int T, bool ABSOLUTE, class Word>
__device__ __forceinline__ uint32_t decode_blocks(Word&& word, uint32_t p, uint32_t blk, const uint32_t end, const uint32_t limit, uint32_t c,
                                                  const uint32_t bpm, const uint32_t luma, ValueMisc<T>& sh, const unsigned char* tab0, int16_t* __restrict__ coef,
                                                  uint32_t* __restrict__ info, uint32_t& err) {
    const uint32_t first = blk;
    if (blk >= end) return 0;
    uint32_t wi = p >> 5;
    uint32_t w0 = word(wi), w1 = word(wi + 1), w2 = word(wi + 2);
    const uint32_t tabs = smem_addr(sh.tabs), tbase = smem_addr(tab0), place = smem_addr(sh.place), buf = smem_addr(&sh.block[threadIdx.x]);
    uint32_t tb = lds32(tabs + c * 4);
    uint32_t tab = tbase + (tb & 0xFFFFu);
    uint32_t z = 0, seen = 0;
    int32_t dc = 0, pred0 = 0, pred1 = 0, pred2 = 0;
    for (;;) {
        const uint32_t top = __funnelshift_l(w1, w0, p);
        uint32_t e = lds32(tab + ((top >> (32 - kLutBits)) << 2));
        if (e == 0) {
            const uint32_t lc = long_code(reinterpret_cast<const LongCodes*>(__cvta_shared_to_generic(tab + (sizeof(uint32_t) << kLutBits))), top);
            if ((lc >> 31) && p < limit) err |= kStBadCode;
            e = huff_pack(lc & 31u, (lc >> 8) & 255u);
        }
        const uint32_t used = e & 63u, len = (e >> 6) & 31u, s = (e >> 11) & 15u, r = (e >> 15) & 15u;
        // the s extra bits (T.81 EXTEND): a leading 1 means the value itself, a leading 0 the complement of its magnitude
        const uint32_t bits = top << len;
        const int32_t neg = ~((int32_t)bits >> 31);
        const int32_t v = (int32_t)(shr_clamp(bits ^ (uint32_t)neg, 32u - s) ^ (uint32_t)neg) - neg;
        p += used;
        if (z == 0) {
            dc = v;
            z = 1;
            tab = tbase + (tb >> 16);
        } else if (s) {
            const uint32_t at = z + r;
            if (at > 63u) { if (p <= limit) err |= kStCoefRange; }
            else {
                const uint32_t pl = lds32(place + at * 4);
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(buf + (pl & 0xFFFFu)), "h"((uint16_t)v) : "memory");
                seen |= pl;
            }
            z = at + 1;
        } else {
            z = r == 15u ? z + 16u : 64u;
        }
        if (z >= 64u) {
            if (p > limit) {  // (what the buffer holds is of no use, and neither is the rest of the span)
                break;
            }
            if (ABSOLUTE) {
                if (c < luma) dc = pred0 += dc;
                else if (c == luma) dc = pred1 += dc;
                else dc = pred2 += dc;
            }
            const uint32_t cls = seen & kNot4x4 ? (uint32_t)kClsFull : seen & kNot2x2 ? (uint32_t)kCls4x4 : seen & kNotDc ? (uint32_t)kCls2x2 : (uint32_t)kClsDc;
            info[blk] = ((uint32_t)dc & 0xFFFFu) | cls << 16;
            uint4* const rows = reinterpret_cast<uint4*>(coef) + (size_t)blk * 8;
            const uint4 zero = make_uint4(0, 0, 0, 0);
            uint4* const b = sh.block + threadIdx.x;
            if (cls <= kCls2x2) {
                rows[0] = b[0]; rows[1] = b[T];
                b[0] = zero; b[T] = zero;
                if (cls <= kCls4x4) {
                    rows[2] = b[2 * T]; rows[3] = b[3 * T];
                    b[2 * T] = zero; b[3 * T] = zero;
                    if (cls == kClsFull) {
#pragma unroll
                        for (int q = 4; q < 8; ++q) { rows[q] = b[q * T]; b[q * T] = zero; }
                    }
                }
            }
            ++blk;
            if (blk >= end) break;
            z = 0; seen = 0;
            c = c + 1 == bpm ? 0u : c + 1;
            tb = lds32(tabs + c * 4);
            tab = tbase + (tb & 0xFFFFu);
        }
        const uint32_t nwi = p >> 5;
        if (nwi != wi) { w0 = w1; w1 = w2; w2 = word(nwi + 2); wi = nwi; }  // a symbol has at most 31 bits: one boundary at a time
    }
    return blk - first;
}

}  // namespace

// ---- restart-free images: one thread per cell -----------------------------------------------------------------------
constexpr int kWriteThreads = (int)kCellsPerCta;
// The CTA's cells are consecutive: their 16 KB of stream are staged in shared memory, a cell per row, rows padded against
// bank conflicts; a block may run 1984 bits (64 symbols of 31 bits) into what follows.
constexpr int kStageRows = kWriteThreads + 3, kStagePitch = (int)kCellBits / 8 + 16;

__global__ void __launch_bounds__(kWriteThreads) k_huff_write(JpegWave w) {
    extern __shared__ __align__(16) unsigned char write_smem[];
    ValueMisc<kWriteThreads>& sh = *reinterpret_cast<ValueMisc<kWriteThreads>*>(write_smem);
    unsigned char* const stage = write_smem + sizeof(ValueMisc<kWriteThreads>);
    unsigned char* const tab0 = stage + kStageRows * kStagePitch;
    const uint32_t o = owner_of(w.write_ctas, blockIdx.x);
    const uint32_t img = w.spec_list[o];
    const JpegDesc& d = w.descs[img];
    const uint32_t cell0 = (blockIdx.x - __ldg(w.write_ctas.first + o)) * kCellsPerCta;
    const uint32_t total = w.us_len[img] * 8u;
    const uint32_t ncell = (total + kCellBits - 1) / kCellBits;
    if (cell0 >= ncell) return;
    const int tid = threadIdx.x;
    {
        constexpr int kPieces = (int)kCellBits / 128;  // 16-byte pieces per row
        const uint8_t* src = w.us + d.us_off + (size_t)cell0 * (kCellBits / 8);
        const uint32_t dst = smem_addr(stage);
        // no further than the stream and its padding reach
        const int rows = (int)min((uint32_t)kStageRows, ncell - cell0 + 2);
        for (int i = tid; i < rows * kPieces; i += kWriteThreads) copy16(dst + (i / kPieces) * kStagePitch + (i % kPieces) * 16, src + (size_t)i * 16);
        copy_commit();
    }
    value_setup<kWriteThreads>(w, d, sh, tab0);
    const uint32_t k = cell0 + tid;
    const uint2* recs = w.cells + d.cell_off;
    uint2 a = make_uint2(0, 0);
    uint32_t b1 = 0;
    if (k < ncell) {
        a = recs[k];
        b1 = min(recs[k + 1].y, d.nblocks);
    }
    copy_wait<0>();
    __syncthreads();
    if (k >= ncell || a.y >= b1) return;
    uint32_t err = 0;
    const uint32_t sbase = smem_addr(stage), word0 = cell0 * (kCellBits / 32);
    auto word = [&](uint32_t i) {
        const uint32_t l = min(i - word0, kStageRows * (kCellBits / 32) - 1u);  // (consistent cells never reach past the stage)
        return lds32(sbase + (l + (l / (kCellBits / 32)) * 4) * 4);
    };
    decode_blocks<kWriteThreads, false>(word, a.x, a.y, b1, total, a.y % d.bpm, d.bpm, d.hs * d.vs, sh, tab0,
                                        w.coef + d.block_off * 64, w.diff + d.block_off, err);
    if (err) atomicOr(w.status + d.item, err);
}

// ---- restart-interval images: one thread per segment -----------------------------------------------------------------
// A segment's first MCU and the zero DC predictors are known, so one pass does it.  The segments of a CTA are consecutive
// in one image; the stream under them is staged when it fits (it does for intervals of a few MCUs), else read in place.
constexpr int kRestartThreads = (int)kSegsPerCta;
constexpr uint32_t kRestartStage = 16384;

__global__ void __launch_bounds__(kRestartThreads) k_huff_restart(JpegWave w) {
    extern __shared__ __align__(16) unsigned char restart_smem[];
    ValueMisc<kRestartThreads>& sh = *reinterpret_cast<ValueMisc<kRestartThreads>*>(restart_smem);
    unsigned char* const stage = restart_smem + sizeof(ValueMisc<kRestartThreads>);
    unsigned char* const tab0 = stage + kRestartStage;
    const uint32_t o = owner_of(w.restart_ctas, blockIdx.x);
    const uint32_t img = w.restart_list[o];
    const JpegDesc& d = w.descs[img];
    const uint32_t k0 = (blockIdx.x - __ldg(w.restart_ctas.first + o)) * kSegsPerCta;
    const int tid = threadIdx.x;
    const uint32_t found = w.seg_found[img], us_len = w.us_len[img], k = k0 + tid;
    if (k0 == 0 && tid == 0 && found != d.nseg) atomicOr(w.status + d.item, kStBadMarker);
    const uint32_t* seg = w.seg_start + d.seg_off;
    const uint32_t have = min(found, d.nseg);  // entries of seg[] that exist
    if (k0 >= have) return;
    // the CTA's piece of the stream: from the 16-byte piece its first segment starts in to its end plus what a block that
    // is not whole may run over
    const uint32_t lo = seg[k0] & ~15u, hi = (k0 + kSegsPerCta < have ? seg[k0 + kSegsPerCta] : us_len) + 272u;
    const bool staged = hi - lo <= kRestartStage;
    const uint8_t* us = w.us + d.us_off;
    if (staged) {
        const uint32_t dst = smem_addr(stage);
        for (uint32_t i = tid; i * 16 < hi - lo; i += kRestartThreads) copy16(dst + i * 16, us + lo + (size_t)i * 16);
        copy_commit();
    }
    value_setup<kRestartThreads>(w, d, sh, tab0);
    copy_wait<0>();
    __syncthreads();
    if (k >= have) return;
    const uint32_t b0 = seg[k], b1 = k + 1 < have ? seg[k + 1] : us_len;
    const uint32_t mcus = d.mcux * d.mcuy;
    const uint32_t m0 = k * d.restart, m1 = min(m0 + d.restart, mcus);
    const uint32_t blk0 = m0 * d.bpm, blk1 = m1 * d.bpm;
    int16_t* coef = w.coef + d.block_off * 64;
    uint32_t* info = w.info + d.block_off;
    uint32_t err = 0, n;
    if (staged) {
        const uint32_t sbase = smem_addr(stage) - lo;
        n = decode_blocks<kRestartThreads, true>([&](uint32_t i) { return lds32(sbase + i * 4); }, b0 * 8u, blk0, blk1, b1 * 8u, 0u, d.bpm,
                                                 d.hs * d.vs, sh, tab0, coef, info, err);
    } else {
        const uint32_t* words = reinterpret_cast<const uint32_t*>(us);
        const uint32_t nwords = (us_len + 3) / 4 + 2;
        n = decode_blocks<kRestartThreads, true>([&](uint32_t i) { return i < nwords ? __ldg(words + i) : 0u; }, b0 * 8u, blk0, blk1, b1 * 8u, 0u,
                                                 d.bpm, d.hs * d.vs, sh, tab0, coef, info, err);
    }
    if (n < blk1 - blk0) err |= kStTruncated;
    if (err) atomicOr(w.status + d.item, err);
}

// ---------------------------------------------------------------------------------------------------------------
// K1b  DC prediction of restart-free images: diff[] holds what info[] will hold, with DC differences, in scan order; the
//      predictor runs over the blocks of a component.  Kept out of the bit-serial kernels on purpose: there it would cost every symbol of the
//      synchronising pass a value extraction, here it is a prefix sum over four bytes per block.
//      One CTA per kDcMcus MCUs of an image; it adds up what lies before its range itself (L2 reads, 32 ranges at most for a
//      50-megapixel image), so that no CTA waits on another.
// ---------------------------------------------------------------------------------------------------------------
namespace {

constexpr int kDcThreads = 512;
struct Dc3 { int32_t a, b, c; };
__device__ __forceinline__ Dc3 operator+(Dc3 x, Dc3 y) { return {x.a + y.a, x.b + y.b, x.c + y.c}; }

// four MCUs per thread: BPM 16-byte pieces
template <int BPM>
__device__ __forceinline__ Dc3 load_mcus(const uint32_t* diff, uint32_t m4, uint32_t nblocks, uint32_t (&v)[4 * BPM]) {
    const uint32_t b0 = m4 * 4 * BPM;
    if (b0 + 4 * BPM <= nblocks) {
#pragma unroll
        for (int i = 0; i < BPM; ++i) {
            const uint4 q = reinterpret_cast<const uint4*>(diff + b0)[i];
            v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4 * BPM; ++i) v[i] = b0 + i < nblocks ? diff[b0 + i] : 0u;
    }
    Dc3 s{0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4 * BPM; ++i) {
        const int k = i % BPM;
        const int32_t x = (int32_t)(int16_t)(v[i] & 0xFFFFu);
        if (BPM == 1 || k < BPM - 2) s.a += x;
        else if (k == BPM - 2) s.b += x;
        else s.c += x;
    }
    return s;
}

template <int BPM>
__device__ void dc_range(const uint32_t* diff, uint32_t* info, uint32_t range, uint32_t nblocks, Dc3* s_warp) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr uint32_t kStep = kDcThreads;  // groups of four MCUs per turn
    const uint32_t groups = (nblocks + 4 * BPM - 1) / (4 * BPM);
    const uint32_t g0 = range * (kDcMcus / 4), g1 = min(g0 + kDcMcus / 4, groups);
    uint32_t v[4 * BPM];
    Dc3 before{0, 0, 0};
    for (uint32_t g = tid; g < g0; g += kStep) before = before + load_mcus<BPM>(diff, g, nblocks, v);
    auto total = [&](Dc3 x) -> Dc3 {  // sum over the CTA, in every thread
#pragma unroll
        for (int o = 16; o; o >>= 1) { x.a += __shfl_xor_sync(0xFFFFFFFFu, x.a, o); x.b += __shfl_xor_sync(0xFFFFFFFFu, x.b, o); x.c += __shfl_xor_sync(0xFFFFFFFFu, x.c, o); }
        __syncthreads();
        if (lane == 0) s_warp[warp] = x;
        __syncthreads();
        Dc3 t{0, 0, 0};
#pragma unroll
        for (int i = 0; i < kDcThreads / 32; ++i) t = t + s_warp[i];
        return t;
    };
    Dc3 carry{0, 0, 0};
    if (g0) carry = total(before);
    // (info keeps 16 bits, so nothing is lost when a damaged stream makes the sums wrap)
    for (uint32_t g = g0; g < g1; g += kStep) {
        const uint32_t m4 = g + tid;
        Dc3 mine{0, 0, 0};
        if (m4 < g1) mine = load_mcus<BPM>(diff, m4, nblocks, v);
        Dc3 inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t ta = __shfl_up_sync(0xFFFFFFFFu, inc.a, o), tb = __shfl_up_sync(0xFFFFFFFFu, inc.b, o), tc = __shfl_up_sync(0xFFFFFFFFu, inc.c, o);
            if (lane >= o) { inc.a += ta; inc.b += tb; inc.c += tc; }
        }
        __syncthreads();
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        Dc3 pre{0, 0, 0}, all{0, 0, 0};
#pragma unroll
        for (int i = 0; i < kDcThreads / 32; ++i) { const Dc3 t = s_warp[i]; if (i < warp) pre = pre + t; all = all + t; }
        int32_t a = carry.a + pre.a + inc.a - mine.a, b = carry.b + pre.b + inc.b - mine.b, c = carry.c + pre.c + inc.c - mine.c;
        carry = carry + all;
        if (m4 >= g1) continue;
        // running predictors; the class bits stay
        const uint32_t b0 = m4 * 4 * BPM;
#pragma unroll
        for (int i = 0; i < 4 * BPM; ++i) {
            const int k = i % BPM;
            const int32_t x = (int32_t)(int16_t)(v[i] & 0xFFFFu);
            int32_t& pred = (BPM == 1 || k < BPM - 2) ? a : k == BPM - 2 ? b : c;
            pred += x;
            v[i] = (v[i] & 0xFFFF0000u) | ((uint32_t)pred & 0xFFFFu);
        }
        if (b0 + 4 * BPM <= nblocks) {
#pragma unroll
            for (int i = 0; i < BPM; ++i) reinterpret_cast<uint4*>(info + b0)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4 * BPM; ++i) if (b0 + i < nblocks) info[b0 + i] = v[i];
        }
    }
}

}  // namespace

__global__ void __launch_bounds__(kDcThreads) k_dc(JpegWave w) {
    __shared__ Dc3 s_warp[kDcThreads / 32];
    const uint32_t o = owner_of(w.dc_ctas, blockIdx.x);
    const JpegDesc& d = w.descs[w.spec_list[o]];
    const uint32_t range = blockIdx.x - __ldg(w.dc_ctas.first + o);
    const uint32_t* diff = w.diff + d.block_off;
    uint32_t* info = w.info + d.block_off;
    switch (d.bpm) {
        case 1: dc_range<1>(diff, info, range, d.nblocks, s_warp); break;
        case 3: dc_range<3>(diff, info, range, d.nblocks, s_warp); break;
        case 4: dc_range<4>(diff, info, range, d.nblocks, s_warp); break;
        default: dc_range<6>(diff, info, range, d.nblocks, s_warp); break;
    }
}

// Stage-by-stage parity tests look at whole coefficient blocks: fills in the rows the class left out and the DC term.
__global__ void __launch_bounds__(256) k_whole_blocks(JpegWave w, uint32_t nblocks) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x, blk = i >> 3, row = i & 7u;
    if (blk >= nblocks) return;
    const uint32_t v = w.info[blk];
    uint4* const at = reinterpret_cast<uint4*>(w.coef) + (size_t)blk * 8 + row;
    uint4 q = row < class_rows((int)(v >> 16 & 3u)) ? *at : make_uint4(0, 0, 0, 0);
    if (row == 0) q.x = (q.x & 0xFFFF0000u) | (v & 0xFFFFu);
    *at = q;
}

// ---- launches -----------------------------------------------------------------------------------------------------------
namespace {

template <class K>
void allow_smem(K kernel, size_t bytes) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); }

// Dynamic shared memory beyond the default limit has to be allowed once per device and kernel.
void configure_once() {
    static std::once_flag done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    std::call_once(done[dev], [] {
        const size_t most = 227 * 1024 - 1024;
        allow_smem(k_huff_sync<256, false>, most);
        allow_smem(k_huff_sync<512, false>, most);
        allow_smem(k_huff_sync<1024, false>, most);
        allow_smem(k_huff_sync<1024, true>, most);
        allow_smem(k_huff_write, most);
        allow_smem(k_huff_restart, most);
    });
}

template <int T, bool CLUSTER>
void launch_sync(const JpegWave& w, uint32_t first, uint32_t count, uint32_t cluster, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(count * cluster);
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = (size_t)T * kRingPitch + sizeof(SyncMisc<T>) + w.max_tables * sizeof(SyncTab);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    if (CLUSTER) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = cluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
    cudaLaunchKernelEx(&cfg, k_huff_sync<T, CLUSTER>, w, first);
}

}  // namespace

// How many threads an image gets.  With hundreds of images in a launch the images fill the GPU by themselves and 256
// threads each (runs of a dozen cells) waste the least on synchronisation; with fewer, an image gets more threads, so
// that the launch does not last as long as one thread's run; with a few tens or less, a cluster of up to eight 1024-thread
// CTAs.  longest_cells: cells of the longest image of the launch (more CTAs than it has cells for would idle).  widest: the
// images are the few longest of a wave, launched beside the others: 1024 threads at least.
void launch_huff_sync(const JpegWave& w, uint32_t first, uint32_t count, uint32_t longest_cells, bool widest, cudaStream_t s) {
    if (!count) return;
    configure_once();
    if (!widest && count >= 3 * 148) { launch_sync<256, false>(w, first, count, 1, s); return; }
    if (!widest && count >= 120) { launch_sync<512, false>(w, first, count, 1, s); return; }
    uint32_t cluster = 1;
    while (cluster < 8 && 2 * cluster * count <= 148 && cluster * 1024 < longest_cells) cluster *= 2;
    if (cluster == 1) launch_sync<1024, false>(w, first, count, 1, s);
    else launch_sync<1024, true>(w, first, count, cluster, s);
}

void launch_huff_write(const JpegWave& w, cudaStream_t s) {
    if (!w.write_ctas.total) return;
    configure_once();
    const size_t smem = sizeof(ValueMisc<kWriteThreads>) + (size_t)kStageRows * kStagePitch + w.max_tables * sizeof(ValueTab);
    k_huff_write<<<w.write_ctas.total, kWriteThreads, smem, s>>>(w);
    k_dc<<<w.dc_ctas.total, kDcThreads, 0, s>>>(w);
}

void launch_huff_restart(const JpegWave& w, cudaStream_t s) {
    if (!w.restart_ctas.total) return;
    configure_once();
    const size_t smem = sizeof(ValueMisc<kRestartThreads>) + kRestartStage + w.max_tables * sizeof(ValueTab);
    k_huff_restart<<<w.restart_ctas.total, kRestartThreads, smem, s>>>(w);
}

void launch_whole_blocks(const JpegWave& w, uint32_t nblocks, cudaStream_t s) {
    if (nblocks) k_whole_blocks<<<(nblocks + 31) / 32, 256, 0, s>>>(w, nblocks);
}

}  // namespace dg
