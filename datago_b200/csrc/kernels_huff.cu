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

#include <cstddef>
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

// ---- code tables ---------------------------------------------------------------------------------------------------------
namespace {

constexpr uint32_t kNoState = 0xFFFFFFFFu;  // "the stream has ended" in place of a bit position

// Codes longer than the fast part of the host's table.  No search: the code length follows from six comparisons against
// the table's left-aligned limits, the symbol from the canonical offset of that length.  v: the next 16 bits.
// Returns length | symbol << 8; 16 with bit 31 set when no code matches.
__device__ __forceinline__ uint32_t long_code(const HuffTable* t, uint32_t v) {
    const uint4 la = __ldg(reinterpret_cast<const uint4*>(&t->limit[0])), lb = __ldg(reinterpret_cast<const uint4*>(&t->limit[4]));
    const uint32_t len = 10u + (v >= la.x) + (v >= la.y) + (v >= la.z) + (v >= la.w) + (v >= lb.x) + (v >= lb.y);
    if (v >= lb.z) return 16u | 0x80000000u;
    return len | ((uint32_t)__ldg(t->vals + (int32_t)(v >> (16u - len)) + __ldg(t->valoff + len)) << 8);
}
// any code at the head of the 16 bits v, same result
__device__ __forceinline__ uint32_t code_at(const HuffTable* t, uint32_t v) {
    const uint32_t e = __ldg(t->lut + (v >> (16 - kLutBits)));
    if (!e) return long_code(t, v);
    return ((e >> 6) & 31u) | ((e >> 11) & 255u) << 8;
}
__device__ __forceinline__ uint32_t advance_of(uint32_t symbol, bool is_ac) {  // slots a symbol advances
    const uint32_t s = symbol & 15u, r = symbol >> 4;
    return !is_ac ? 1u : (s || r == 15u) ? r + 1u : 64u;  // coefficient after a run, ZRL, or end of block
}

// Look-up tables of the two decoders for one (DC, AC) pair of Huffman tables, made on the device (k_unstuff_count), because
// they are several times the size of what the host sends.  Codes longer than the index: entry 0, and far[] takes over --
// canonical codes grow with their length, so all of them lie above far_base, and the 16-bit windows from there on are few
// (190 to 640 for the tables most files carry).  Windows behind the end of far[] go to the host's table.
constexpr int kSyncBits = 10, kValueBits = 9;
// Synchronising decoder: as many whole symbols as the index shows.  bits 0-4 / 5-11: bits consumed and slots advanced by the
// first symbol alone, 12-16 / 17-23: by all of them, 24-29: slots before the last one (the last counts only if that many do
// not end the block).  64 slots or more end the block.  A DC symbol is followed by AC symbols of the same component.
struct SyncTab {
    uint32_t lut[1 << kSyncBits];
    uint32_t far[384];
    uint32_t far_base, huff, is_ac, pad;
};
// Value decoder: bits 0-4 code and extra bits together, 5-9 code length, 10-13 extra bits s, 24 no such code, 25-31 slots
// advanced (the coefficient sits in the last of them; 64: end of block).
struct ValueTab {
    uint32_t lut[1 << kValueBits];
    uint32_t far[640];
    uint32_t far_base, huff, is_ac, pad;
};
struct CodeTables { SyncTab sync[2]; ValueTab value[2]; };  // [0] DC, [1] AC
static_assert(sizeof(SyncTab) % 16 == 0 && sizeof(ValueTab) % 16 == 0 && sizeof(CodeTables) == kCodeTablesBytes, "tables are copied in 16-byte pieces");

__device__ __forceinline__ uint32_t sync_entry(uint32_t u, uint32_t a) { return u | a << 5 | u << 12 | a << 17; }
__device__ __forceinline__ uint32_t value_entry(uint32_t code, bool is_ac) {
    const uint32_t len = code & 31u, s = (code >> 8) & 15u;
    return (len + s) | len << 5 | s << 10 | (code >> 31) << 24 | advance_of((code >> 8) & 255u, is_ac) << 25;
}

__device__ void build_tables(CodeTables& out, const HuffTable* pool, uint32_t dc_id, uint32_t ac_id, int tid, int nthreads) {
    const HuffTable* const ac = pool + ac_id;
    for (int side = 0; side < 2; ++side) {
        const HuffTable* const t = pool + (side ? ac_id : dc_id);
        SyncTab& st = out.sync[side];
        ValueTab& vt = out.value[side];
        for (uint32_t i = tid; i < (1u << kSyncBits); i += nthreads) {
            const uint32_t window = i << (16 - kSyncBits);
            uint32_t c = code_at(t, window), e = 0;
            if ((c & 31u) <= (uint32_t)kSyncBits) {
                uint32_t u = (c & 31u) + ((c >> 8) & 15u), a = advance_of((c >> 8) & 255u, side != 0), pre = 0;
                const uint32_t first = u | a << 5;
                while (u < (uint32_t)kSyncBits && a < 64u) {
                    c = code_at(ac, (window << u) & 0xFFFFu);
                    const uint32_t len = c & 31u;
                    if (u + len > (uint32_t)kSyncBits) break;
                    pre = a;
                    u += len + ((c >> 8) & 15u);
                    a += advance_of((c >> 8) & 255u, true);
                }
                e = first | u << 12 | a << 17 | pre << 24;
            }
            st.lut[i] = e;
        }
        // the windows from the first one that no code of at most kLutBits / kSyncBits bits covers
        uint32_t covered = 0;
        for (int k = 0; k < (1 << kLutBits); k += 32) covered += __popc(__ballot_sync(0xFFFFFFFFu, __ldg(t->lut + k + (tid & 31)) != 0u));
        const uint32_t vbase = covered << (16 - kLutBits), sbase = __ldg(t->limit + 0);
        static_assert(kValueBits == kLutBits && kSyncBits == 10, "limit[0] covers ten bits");
        for (uint32_t i = tid; i < sizeof(st.far) / 4; i += nthreads) {
            const uint32_t c = code_at(t, min(sbase + i, 0xFFFFu));
            st.far[i] = sync_entry((c & 31u) + ((c >> 8) & 15u), advance_of((c >> 8) & 255u, side != 0));
        }
        for (uint32_t i = tid; i < (1u << kValueBits); i += nthreads) {
            const uint32_t c = code_at(t, i << (16 - kValueBits));
            vt.lut[i] = (c & 31u) <= (uint32_t)kValueBits ? value_entry(c, side != 0) : 0u;
        }
        for (uint32_t i = tid; i < sizeof(vt.far) / 4; i += nthreads) vt.far[i] = value_entry(code_at(t, min(vbase + i, 0xFFFFu)), side != 0);
        if (tid == 0) {
            st.far_base = sbase; vt.far_base = vbase;
            st.huff = vt.huff = side ? ac_id : dc_id;
            st.is_ac = vt.is_ac = side;
        }
    }
}

// the entry of a code longer than the index; `tab`: shared-memory address of the table
template <class Tab>
__device__ __forceinline__ uint32_t far_entry(uint32_t tab, uint32_t top, const HuffTable* pool) {
    const uint32_t v = top >> 16, i = v - lds32(tab + (uint32_t)offsetof(Tab, far_base));
    if (i < (uint32_t)(sizeof(Tab::far) / 4)) return lds32(tab + (uint32_t)offsetof(Tab, far) + i * 4);
    const uint32_t c = long_code(pool + lds32(tab + (uint32_t)offsetof(Tab, huff)), v);
    const bool is_ac = lds32(tab + (uint32_t)offsetof(Tab, is_ac)) != 0;
    if (sizeof(Tab) == sizeof(SyncTab)) return sync_entry((c & 31u) + ((c >> 8) & 15u), advance_of((c >> 8) & 255u, is_ac));
    return value_entry(c, is_ac);
}

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

// (The CTAs behind the last tile make the code tables of the wave: work of the same length, for which a launch of its own
// would be too much.)
__global__ void __launch_bounds__(kUnstuffThreads) k_unstuff_count(JpegWave w) {
    if (blockIdx.x >= w.us_tiles.total) {
        const uint32_t k = blockIdx.x - w.us_tiles.total;
        const uint2 ids = w.table_pairs[k];
        build_tables(reinterpret_cast<CodeTables*>(w.codes)[k], w.huff, ids.x, ids.y, threadIdx.x, kUnstuffThreads);
        return;
    }
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
    k_unstuff_count<<<w.us_tiles.total + w.n_pairs, kUnstuffThreads, 0, s>>>(w);
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

// Where a decoder stands inside the MCU: the tables of the current block as shared-memory addresses, and the entry of the
// block after it.  One 16-byte read per block instead of arithmetic on indices.
struct McuBlock { uint32_t dc, ac, next, index; };
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// The image's tables into shared memory, each distinct pair once.  Tab: SyncTab or ValueTab; which: offset of its [2] array
// inside CodeTables.
template <class Tab>
__device__ __forceinline__ void load_tables(const JpegWave& w, const JpegDesc& d, McuBlock* mcu, unsigned char* tab0, uint32_t which, int tid, int nthreads) {
    const uint32_t p0 = d.pair[0], p1 = d.pair[1], p2 = d.pair[2];
    const uint32_t slot1 = p1 == p0 ? 0u : 1u, slot2 = p2 == p0 ? 0u : p2 == p1 ? slot1 : slot1 + 1u;
    constexpr uint32_t kPieces = 2 * sizeof(Tab) / 16;
    const uint32_t nslot = max(slot1, slot2) + 1u;
    for (uint32_t k = 0; k < nslot; ++k) {
        const uint32_t id = k == 0 ? p0 : k == slot1 ? p1 : p2;
        const uint4* src = reinterpret_cast<const uint4*>(w.codes + (size_t)id * kCodeTablesBytes + which);
        const uint32_t dst = smem_addr(tab0) + k * 2 * (uint32_t)sizeof(Tab);
        for (uint32_t i = tid; i < kPieces; i += nthreads) copy16(dst + i * 16, src + i);
    }
    if ((uint32_t)tid < d.bpm) {
        const uint32_t luma = d.hs * d.vs, slot = (uint32_t)tid < luma ? 0u : (uint32_t)tid == luma ? slot1 : slot2;
        const uint32_t at = smem_addr(tab0) + slot * 2 * (uint32_t)sizeof(Tab);
        mcu[tid] = McuBlock{at, at + (uint32_t)sizeof(Tab), smem_addr(&mcu[(uint32_t)tid + 1 == d.bpm ? 0 : tid + 1]), (uint32_t)tid};
    }
}

// Window of two stream words (w0 holds the current bit): when bit position `was` -> `now` crosses a word boundary (one at
// most: symbols have 31 bits at most), w0 takes w1 and w1 the word behind the one at address `word`.  Predicated by hand:
// some lane of a warp crosses in nearly every step.
__device__ __forceinline__ void advance_window(uint32_t& w0, uint32_t& w1, uint32_t was, uint32_t now, uint32_t word) {
    asm volatile("{\n .reg .pred q;\n setp.ge.u32 q, %2, 32;\n @q mov.u32 %0, %1;\n @q ld.shared.u32 %1, [%3+4];\n}" : "+r"(w0), "+r"(w1) : "r"(was ^ now), "r"(word));
}
// Streams in shared memory: at(p) is the address of the word that holds bit p; the word behind it follows.
template <class Address>
struct SharedSource {
    Address at;
    __device__ __forceinline__ void start(uint32_t& w0, uint32_t& w1, uint32_t p) const { w0 = lds32(at(p)); w1 = lds32(at(p) + 4); }
    __device__ __forceinline__ void advance(uint32_t& w0, uint32_t& w1, uint32_t was, uint32_t now) const { advance_window(w0, w1, was, now, at(now)); }
};
template <class Address> __device__ __forceinline__ SharedSource<Address> shared_source(Address at) { return SharedSource<Address>{at}; }
// ... and in global memory
struct GlobalSource {
    const uint32_t* words;
    uint32_t n;
    __device__ __forceinline__ uint32_t word(uint32_t i) const { return i < n ? __ldg(words + i) : 0u; }
    __device__ __forceinline__ void start(uint32_t& w0, uint32_t& w1, uint32_t p) const { w0 = word(p >> 5); w1 = word((p >> 5) + 1); }
    __device__ __forceinline__ void advance(uint32_t& w0, uint32_t& w1, uint32_t was, uint32_t now) const {
        if ((was ^ now) >= 32u) { w0 = w1; w1 = word((now >> 5) + 1); }
    }
};

// A lane of a synchronising decoder.
struct SyncLane {
    uint32_t p, z, nb;   // bit position, slot inside the block, blocks ended since nb was last set to zero
    uint32_t w0, w1, tab;
    uint4 mb;            // McuBlock of the current block
    template <class Source>
    __device__ __forceinline__ void start(const Source& src, uint32_t mcu0, uint32_t bit, uint32_t slot, uint32_t c) {
        p = bit; z = slot; nb = 0;
        src.start(w0, w1, p);
        mb = lds128(mcu0 + c * (uint32_t)sizeof(McuBlock));
        tab = z ? mb.y : mb.x;
    }
    // Lanes with `live` decode to the first block start at p >= stop.  Called by whole warps: the loop has one exit, taken by
    // all lanes together, and no other jump out of it -- with returns from inside, the lanes of a warp never met again
    // after their first different turn and went on alone.  turn(): called every four steps (124 bits at most) by all.
    template <class Source, class Turn>
    __device__ __forceinline__ void run_to(bool live, uint32_t stop, const Source& src, const HuffTable* pool, Turn&& turn) {
        while (__any_sync(0xFFFFFFFFu, live)) {
            turn(live);
#pragma unroll
            for (int step = 0; step < 4; ++step) {
                if (live) {
                    const uint32_t top = __funnelshift_l(w1, w0, p);
                    uint32_t e = lds32(tab + ((top >> (32 - kSyncBits)) << 2));
                    if (e == 0) e = far_entry<SyncTab>(tab, top, pool);
                    const uint32_t h = z + (e >> 24) >= 64u ? e : e >> 12;
                    const uint32_t was = p;
                    p += h & 31u;
                    z += (h >> 5) & 127u;
                    tab = mb.y;
                    src.advance(w0, w1, was, p);
                    if (z >= 64u) {
                        z = 0;
                        ++nb;
                        mb = lds128(mb.z);
                        tab = mb.x;
                        live = p < stop;
                    }
                }
            }
        }
    }
};

constexpr int kRingPitch = 144;  // bytes per thread: eight 16-byte pieces of its stream, and the first of them once more behind them

template <int T>
struct SyncMisc {
    uint2 exit[T];         // state each thread hands to its right neighbour
    McuBlock mcu[6];
    uint32_t warp[32];
    uint32_t flag[3];      // cluster: some thread still differs (by round, modulo 3)
    uint32_t total;        // blocks found by this CTA's threads
    uint32_t pad[3];
};
static_assert(sizeof(SyncMisc<256>) % 16 == 0, "tables follow in shared memory");

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
    load_tables<SyncTab>(w, d, sh.mcu, tab0, (uint32_t)offsetof(CodeTables, sync), tid, T);
    copy_commit();
    if (tid < 3) sh.flag[tid] = 0;
    copy_wait<0>();
    __syncthreads();

    const uint32_t total = w.us_len[img] * 8u;
    const uint32_t ncell = (total + kCellBits - 1) / kCellBits;
    const uint8_t* const us = w.us + d.us_off;
    uint2* const recs = w.cells + d.cell_off;
    const uint32_t gt = rank * T + tid, nthread = nrank * T;
    const uint32_t run = (ncell + nthread - 1) / nthread;
    const uint32_t kbeg = min(gt * run, ncell), kend = min(kbeg + run, ncell);
    const bool active = kbeg < kend;
    const uint32_t ring = smem_addr(ring0) + tid * kRingPitch, mcu0 = smem_addr(&sh.mcu[0]);

    uint32_t found = 0;                       // blocks that start in this thread's cells
    uint2 entry = make_uint2(0, 0), exit = make_uint2(kNoState, 0);

    // Decodes the thread's cells from (p, z, c).  Redoing, it stops as soon as it meets the state recorded for one of them.
    auto decode = [&](bool live, uint32_t p, uint32_t z, uint32_t c, bool redo) {
        // the stream in pieces of 16 bytes through this thread's ring
        const bool ended = p == kNoState;
        uint32_t wr = ended ? 0u : p >> 7;
        SyncLane L;
        L.p = p;
        auto fetch = [&]() {
            copy16(ring + (wr & 7u) * 16, us + (size_t)wr * 16);
            if ((wr & 7u) == 0) copy16(ring + 128, us + (size_t)wr * 16);
            ++wr;
        };
        if (live && !ended) {
            for (int i = 0; i < 8; ++i) fetch();
        }
        copy_commit();
        copy_wait<0>();
        const auto source = shared_source([&](uint32_t bit) { return ring + ((bit >> 3) & 124u); });
        // A step consumes at most 31 bits, so four of them cross at most one piece and one copy per turn keeps the ring
        // full.  The copies of the last four turns may still be under way: they are at least three pieces ahead.
        auto turn = [&](bool on) {
            if (on && wr < (L.p >> 7) + 8) fetch();
            copy_commit();
            copy_wait<4>();
        };
        L.start(source, mcu0, p, z, c);
        if (!redo) L.run_to(live && z != 0, kbeg * kCellBits, source, w.huff, turn);  // the guess: to the first block start it meets
        for (uint32_t i = 0; i < run; ++i) {
            const uint32_t k = kbeg + i, bound = (k + 1) * kCellBits;
            bool on = live && k < kend;
            if (L.p > total) { L.p = kNoState; L.mb.w = 0; }  // the block that ended here is not whole
            const uint2 at = make_uint2(L.p, L.mb.w);
            uint32_t old_n = 0;
            if (on) {
                if (redo) {
                    const uint2 had = recs[k];
                    old_n = had.y & 0x0FFFFFFFu;
                    if (i && had.x == at.x && (had.y >> 28) == at.y) on = live = false;  // met
                }
                if (!redo && i == 0) entry = at;
            }
            if (!__any_sync(0xFFFFFFFFu, on)) break;
            L.nb = 0;
            L.run_to(on && L.p < bound, min(bound, total + 1), source, w.huff, turn);
            if (on) {
                if (L.p > total && L.p != kNoState) --L.nb;
                recs[k] = make_uint2(at.x, at.y << 28 | L.nb);
                found += L.nb - old_n;
            }
        }
        // Nothing may be on its way into the ring when it is filled anew: of two copies to one place the older may land last.
        copy_wait<0>();
        if (L.p > total) { L.p = kNoState; L.mb.w = 0; }
        if (live) exit = make_uint2(L.p, L.mb.w);
    };

    decode(active, gt ? kbeg * kCellBits : 0u, gt ? 1u : 0u, 0u, false);
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
        if (__any_sync(0xFFFFFFFFu, need)) {
            decodes += need;
            if (need) entry = prev;
            decode(need, need ? prev.x : kNoState, 0, prev.y, true);
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

constexpr uint32_t kNotDc = 1u << 28, kNot2x2 = 1u << 29, kNot4x4 = 1u << 30;

// Zig-zag position -> byte offset of the coefficient in a lane's block buffer (row r of the lane's block sits at
// r * T * 16: rows of neighbouring lanes are neighbours, so whole-row accesses are conflict free) | class flags.
template <int T>
__device__ __forceinline__ uint32_t place_of(uint32_t zz) {
    const uint32_t nat = kNatural[zz], r = nat >> 3, c = nat & 7u;
    return r * (T * 16) + c * 2 | (zz ? kNotDc : 0u) | (r > 1 || c > 1 ? kNot2x2 : 0u) | (r > 3 || c > 3 ? kNot4x4 : 0u);
}

template <int T>
struct ValueMisc {
    uint4 block[8 * T];    // the lanes' current blocks
    uint32_t place[64];
    McuBlock mcu[6];
    uint32_t pad[8];
};

// Shared memory of the value decoder: [ValueMisc | ... | tables].  The caller waits for the copies and the barrier.
template <int T>
__device__ __forceinline__ void value_setup(const JpegWave& w, const JpegDesc& d, ValueMisc<T>& sh, unsigned char* tab0) {
    const int tid = threadIdx.x;
    load_tables<ValueTab>(w, d, sh.mcu, tab0, (uint32_t)offsetof(CodeTables, value), tid, T);
    copy_commit();
    if (tid < 64) sh.place[tid] = place_of<T>(tid);
#pragma unroll
    for (int r = 0; r < 8; ++r) sh.block[r * T + tid] = make_uint4(0, 0, 0, 0);
}

// Decodes blocks [blk, end) of an image from bit p on.  src: the image's stream, see SharedSource.
// limit: blocks that reach beyond this bit are not whole -- decoding stops there; so it does at a block that starts at or
// behind `stop`.  ABSOLUTE: the DC predictors start at zero here (a restart segment) and info[] receives the DC terms
// themselves instead of their differences.  Returns the blocks decoded.  Called by whole warps.
//
// One code path for DC and AC symbols, the DC difference going to slot 0 of the block buffer like any coefficient: the lanes
// of a warp are at unrelated places.  For the same reason a lane whose block is complete waits until kFlushLanes lanes
// have one (or no lane has anything else to do): writing a block out takes more instructions than decoding a symbol,
// and they cost the same whether two lanes execute them or ten.
constexpr int kFlushLanes = 8;

template <int T, bool ABSOLUTE, class Source>
__device__ __forceinline__ uint32_t decode_blocks(const Source& src, uint32_t p, uint32_t blk, const uint32_t end, const uint32_t limit, const uint32_t stop,
                                                  uint32_t c, const uint32_t luma, ValueMisc<T>& sh, const HuffTable* pool, int16_t* __restrict__ coef,
                                                  uint32_t* __restrict__ info, uint32_t& err) {
    const uint32_t first = blk;
    bool live = blk < end;
    uint32_t w0, w1;
    src.start(w0, w1, p);
    const uint32_t place = smem_addr(sh.place) - 4, buf = smem_addr(&sh.block[threadIdx.x]);
    uint4 mb = lds128(smem_addr(&sh.mcu[0]) + c * sizeof(McuBlock));
    uint32_t tab = mb.x, z = 0, seen = 0;
    int32_t pred0 = 0, pred1 = 0, pred2 = 0;
    for (;;) {
        const uint32_t alive = __ballot_sync(0xFFFFFFFFu, live);
        if (!alive) break;  // one exit for the whole warp, see k_huff_sync
        if (live && z < 64u) {
            const uint32_t top = __funnelshift_l(w1, w0, p);
            uint32_t e = lds32(tab + ((top >> (32 - kValueBits)) << 2));
            if (e == 0) {
                e = far_entry<ValueTab>(tab, top, pool);
                if (((e >> 24) & 1u) && p < limit) err |= kStBadCode;
            }
            const uint32_t was = p, s = (e >> 10) & 15u;
            // the s extra bits (T.81 EXTEND): a leading 1 means the value itself, a leading 0 the complement of its magnitude
            const uint32_t bits = top << ((e >> 5) & 31u);
            const int32_t neg = ~((int32_t)bits >> 31);
            const int32_t v = (int32_t)(shr_clamp(bits ^ (uint32_t)neg, 32u - s) ^ (uint32_t)neg) - neg;
            p += e & 31u;
            z += e >> 25;
            src.advance(w0, w1, was, p);
            if (s && z <= 64u) {
                const uint32_t pl = lds32(place + z * 4);
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(buf + (pl & 0xFFFFu)), "h"((uint16_t)v) : "memory");
                seen |= pl;
            }
            if (s && z > 64u && p <= limit) err |= kStCoefRange;
            tab = mb.y;
        }
        const uint32_t done = __ballot_sync(0xFFFFFFFFu, live && z >= 64u);
        if (__popc(done) >= kFlushLanes || done == alive) {
            if (live && z >= 64u) {
                if (p > limit) live = false;  // (what the buffer holds is of no use, and neither is the rest of the span)
                else {
                    uint4* const b = sh.block + threadIdx.x;
                    uint4* const rows = reinterpret_cast<uint4*>(coef) + (size_t)blk * 8;
                    const uint4 zero = make_uint4(0, 0, 0, 0), q0 = b[0];
                    int32_t dc = (int16_t)(q0.x & 0xFFFFu);
                    if (ABSOLUTE) {
                        if (mb.w < luma) dc = pred0 += dc;
                        else if (mb.w == luma) dc = pred1 += dc;
                        else dc = pred2 += dc;
                    }
                    const uint32_t cls = seen & kNot4x4 ? (uint32_t)kClsFull : seen & kNot2x2 ? (uint32_t)kCls4x4 : seen & kNotDc ? (uint32_t)kCls2x2 : (uint32_t)kClsDc;
                    info[blk] = ((uint32_t)dc & 0xFFFFu) | cls << 16;
                    b[0] = zero;
                    if (cls <= kCls2x2) {
                        rows[0] = q0; rows[1] = b[T];
                        b[T] = zero;
                    }
                    if (cls <= kCls4x4) {
                        rows[2] = b[2 * T]; rows[3] = b[3 * T];
                        b[2 * T] = zero; b[3 * T] = zero;
                    }
                    if (cls == kClsFull) {
#pragma unroll
                        for (int q = 4; q < 8; ++q) { rows[q] = b[q * T]; b[q * T] = zero; }
                    }
                    ++blk;
                    live = blk < end && p < stop;
                    z = 0; seen = 0;
                    mb = lds128(mb.z);
                    tab = mb.x;
                }
            }
        }
    }
    return blk - first;
}

}  // namespace

// ---- restart-free images: one thread per cell -----------------------------------------------------------------------
constexpr int kWriteThreads = (int)kCellsPerCta;
// The CTA's cells are consecutive: their 16 KB of stream are staged in shared memory, a cell per row and the first 16 bytes
// of the next cell behind it (which spreads the rows over the banks and makes the word behind any word its neighbour); a
// block may run 1984 bits (64 symbols of 31 bits) into what follows.
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
        constexpr int kPieces = (int)kCellBits / 128 + 1;  // 16-byte pieces per row
        const uint8_t* src = w.us + d.us_off + (size_t)cell0 * (kCellBits / 8);
        const uint32_t dst = smem_addr(stage);
        // no further than the stream and its padding reach
        const int rows = (int)min((uint32_t)kStageRows, ncell - cell0 + 2);
        for (int i = tid; i < rows * kPieces; i += kWriteThreads) copy16(dst + i * 16, src + (i / kPieces) * (kCellBits / 8) + (i % kPieces) * 16);
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
    uint32_t err = 0;
    const uint32_t sbase = smem_addr(stage) - cell0 * kStagePitch;
    const auto source = shared_source([&](uint32_t p) { return sbase + ((p >> 3) & ~3u) + (p / kCellBits) * 16; });
    const uint32_t p0 = a.y < b1 ? a.x : cell0 * kCellBits;
    decode_blocks<kWriteThreads, false>(source, p0, a.y, b1, total, (cell0 + kCellsPerCta) * kCellBits, a.y % d.bpm, d.hs * d.vs, sh, w.huff,
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
    const bool mine = k < have;
    const uint32_t b0 = mine ? seg[k] : lo, b1 = k + 1 < have ? seg[k + 1] : us_len;
    const uint32_t mcus = d.mcux * d.mcuy;
    const uint32_t m0 = mine ? k * d.restart : 0u, m1 = mine ? min(m0 + d.restart, mcus) : 0u;
    const uint32_t blk0 = m0 * d.bpm, blk1 = m1 * d.bpm;
    int16_t* coef = w.coef + d.block_off * 64;
    uint32_t* info = w.info + d.block_off;
    uint32_t err = 0, n;
    if (staged) {
        const uint32_t sbase = smem_addr(stage) - lo;
        n = decode_blocks<kRestartThreads, true>(shared_source([&](uint32_t p) { return sbase + ((p >> 3) & ~3u); }), b0 * 8u, blk0, blk1, b1 * 8u, b1 * 8u, 0u,
                                                 d.hs * d.vs, sh, w.huff, coef, info, err);
    } else {
        const GlobalSource source{reinterpret_cast<const uint32_t*>(us), (us_len + 3) / 4 + 2};
        n = decode_blocks<kRestartThreads, true>(source, b0 * 8u, blk0, blk1, b1 * 8u, b1 * 8u, 0u, d.hs * d.vs, sh, w.huff, coef, info, err);
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
    cfg.dynamicSmemBytes = (size_t)T * kRingPitch + sizeof(SyncMisc<T>) + w.max_pairs * 2 * sizeof(SyncTab);
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
    const size_t smem = sizeof(ValueMisc<kWriteThreads>) + (size_t)kStageRows * kStagePitch + w.max_pairs * 2 * sizeof(ValueTab);
    k_huff_write<<<w.write_ctas.total, kWriteThreads, smem, s>>>(w);
    k_dc<<<w.dc_ctas.total, kDcThreads, 0, s>>>(w);
}

void launch_huff_restart(const JpegWave& w, cudaStream_t s) {
    if (!w.restart_ctas.total) return;
    configure_once();
    const size_t smem = sizeof(ValueMisc<kRestartThreads>) + kRestartStage + w.max_pairs * 2 * sizeof(ValueTab);
    k_huff_restart<<<w.restart_ctas.total, kRestartThreads, smem, s>>>(w);
}

void launch_whole_blocks(const JpegWave& w, uint32_t nblocks, cudaStream_t s) {
    if (nblocks) k_whole_blocks<<<(nblocks + 31) / 32, 256, 0, s>>>(w, nblocks);
}

}  // namespace dg
