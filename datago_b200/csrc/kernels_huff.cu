// Baseline JPEG entropy decoding on sm_100a: byte unstuffing, Huffman decode, DC prediction.  First half of the decode
// datago reaches through image::load_from_memory (src/worker_wds.rs:45) / ImageReader::decode (src/worker_files.rs:14-16).
//
// Output of this file, per 8x8 block in scan (MCU-interleaved) order:
//   info[block]  low half: the DC coefficient (int16, prediction resolved); bits 16-17: the block's class
//   coef[block]  64 int16 in natural order -- only the rows the class covers are written (and read), and the DC slot holds
//                nothing to rely on: the term is in info[]
// The class says where the AC coefficients end (kClsFull / kCls4x4 / kCls2x2 / kClsDc).  On photographs at ordinary
// qualities half of the blocks or more carry a handful of low-frequency coefficients or none, so keeping the DC terms
// dense and skipping the rows that hold nothing is worth several times the memory traffic of whole blocks, and nothing has
// to be zeroed before or after.
#include <cstddef>
#include <cstdint>
#include <mutex>

#include <cooperative_groups.h>

#include "kernels.h"

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
// slots a symbol advances, or kBlockEnd
constexpr uint32_t kBlockEnd = 128;
__device__ __forceinline__ uint32_t advance_of(uint32_t symbol, bool is_ac) {
    const uint32_t s = symbol & 15u, r = symbol >> 4;
    return !is_ac ? 1u : (s || r == 15u) ? r + 1u : kBlockEnd;  // coefficient after a run, ZRL, or end of block
}

// Look-up tables of the two decoders for one (DC, AC) pair of Huffman tables, made on the device (k_unstuff_count), because
// they are several times the size of what the host sends.  Both decoders are chains of dependent instructions with few
// warps to hide them, so the tables are laid out for as few instructions per symbol as possible:
//   * A lane keeps its place in one register: bits 0-15 the bit position inside the block (relative to a word boundary),
//     16-21 the slot inside the block, 22-23 "the block has ended" (slot 64 reached, or end of block: kBlockEnd).  A symbol
//     adds to both fields at once.
//   * The codes of at most kBits bits fill entries [0, N) by the next kBits bits; the 16-bit windows of longer codes all lie
//     above those (canonical codes grow with their length) and follow from entry N on, window by window.  The index is then
//     the larger of (top >> 32 - kBits) and (top >> 16) + off: both are N at the first long window, and the first grows
//     slower.  No branch and no second look-up for long codes -- some lane of a warp has one in nearly every step.  Windows
//     behind the last entry, which is 0, and (value decoder) codes that do not exist take the host's table: rare_entry.
constexpr int kSyncBits = 10, kValueBits = 9;
// Synchronising decoder: as many whole symbols as the index shows.  byte 0 / 1: bits consumed and slots advanced (kBlockEnd on
// top if the last one ends the block) by all of them, byte 2 / 3: by the first alone.  Where all would reach slot 64, the
// first is taken alone.  A DC symbol is followed by AC symbols of the same component.
struct SyncTab {
    static constexpr int kBits = kSyncBits, kEntries = (1 << kSyncBits) + 384;
    uint32_t entry[kEntries];
    int32_t off;
    uint32_t huff, is_ac, pad;
};
// Value decoder, to be added to a lane's place as it is: bits 0-4 code and extra bits together, 16-23 slots advanced (the
// coefficient sits in the last of them) or kBlockEnd, 27-31 (32 - s) % 32 for s extra bits: negative if there are any.
struct ValueTab {
    static constexpr int kBits = kValueBits, kEntries = (1 << kValueBits) + 640;
    uint32_t entry[kEntries];
    int32_t off;
    uint32_t huff, is_ac, pad;
};
struct CodeTables { SyncTab sync[2]; ValueTab value[2]; };  // [0] DC, [1] AC
static_assert(sizeof(SyncTab) % 16 == 0 && sizeof(ValueTab) % 16 == 0 && sizeof(CodeTables) == kCodeTablesBytes, "tables are copied in 16-byte pieces");
constexpr uint32_t kPosMask = 0xFFFFu, kEndMask = 0xC0u << 16;  // of a lane's place

// code: see long_code
__device__ __forceinline__ uint32_t sync_entry(uint32_t code, bool is_ac) {  // of one symbol
    return ((code & 31u) + ((code >> 8) & 15u) | advance_of((code >> 8) & 255u, is_ac) << 8) * 0x10001u;
}
__device__ __forceinline__ uint32_t value_entry(uint32_t code, bool is_ac) {
    const uint32_t len = code & 31u, s = (code >> 8) & 15u;
    return (len + s) | advance_of((code >> 8) & 255u, is_ac) << 16 | (32u - s) << 27;
}

// One CTA per table: part 0 / 1 sync[0] / sync[1], 2 / 3 value[0] / value[1].  (One CTA for all four took 8 us, twice what the tiles
// beside it take for an ordinary file.)
constexpr uint32_t kTableParts = 4;
__device__ void build_table(CodeTables& out, const HuffTable* pool, uint32_t dc_id, uint32_t ac_id, uint32_t part, int tid, int nthreads) {
    const uint32_t side = part & 1u;
    const HuffTable* const t = pool + (side ? ac_id : dc_id);
    static_assert(kValueBits == kLutBits && kSyncBits == 10, "limit[0] covers ten bits");
    if (part < 2) {
        SyncTab& st = out.sync[side];
        const HuffTable* const ac = pool + ac_id;
        const uint32_t far = __ldg(t->limit + 0), near = far >> (16 - kSyncBits);  // the first window that no code of at most kSyncBits bits covers
        for (uint32_t i = tid; i < (uint32_t)SyncTab::kEntries; i += nthreads) {
            const uint32_t window = i < near ? i << (16 - kSyncBits) : min(far + (i - near), 0xFFFFu);
            uint32_t c = code_at(t, window), e = sync_entry(c, side != 0);
            if (i < near) {
                uint32_t u = e & 31u, a = (e >> 8) & 255u;
                while (u < (uint32_t)kSyncBits && a < 64u) {
                    c = code_at(ac, (window << u) & 0xFFFFu);
                    const uint32_t len = c & 31u, more = advance_of((c >> 8) & 255u, true);
                    if (u + len > (uint32_t)kSyncBits || (more < kBlockEnd && a + more > 63u)) break;
                    u += len + ((c >> 8) & 15u);
                    a += more;
                }
                e = (e & 0xFFFF0000u) | u | a << 8;
            }
            st.entry[i] = i + 1 < (uint32_t)SyncTab::kEntries ? e : 0u;
        }
        if (tid == 0) { st.off = (int32_t)near - (int32_t)far; st.huff = side ? ac_id : dc_id; st.is_ac = side; }
    } else {
        ValueTab& vt = out.value[side];
        uint32_t covered = 0;  // windows of kLutBits bits that start with a code
        for (int k = 0; k < (1 << kLutBits); k += 32) covered += __popc(__ballot_sync(0xFFFFFFFFu, __ldg(t->lut + k + (tid & 31)) != 0u));
        const uint32_t far = covered << (16 - kLutBits), near = far >> (16 - kValueBits);
        for (uint32_t i = tid; i < (uint32_t)ValueTab::kEntries; i += nthreads) {
            const uint32_t c = code_at(t, i < near ? i << (16 - kValueBits) : min(far + (i - near), 0xFFFFu));
            vt.entry[i] = i + 1 < (uint32_t)ValueTab::kEntries && !(c >> 31) ? value_entry(c, side != 0) : 0u;
        }
        if (tid == 0) { vt.off = (int32_t)near - (int32_t)far; vt.huff = side ? ac_id : dc_id; vt.is_ac = side; }
    }
}

// The entry of the code at the head of `top`, 0: see rare_entry.  tab: shared-memory address of the table, off: its `off`.
template <class Tab>
__device__ __forceinline__ uint32_t entry_at(uint32_t tab, int32_t off, uint32_t top) {
    const int32_t i = min(__viaddmax_s32((int32_t)(top >> 16), off, (int32_t)(top >> (32 - Tab::kBits))), Tab::kEntries - 1);
    return lds32(tab + (uint32_t)i * 4u);
}
// ... of a code whose window lies behind the last entry (x), and the code (y; bit 31: there is no such code).
template <class Tab>
__device__ __noinline__ uint2 rare_entry(uint32_t tab, uint32_t top, const HuffTable* pool) {
    const uint32_t c = long_code(pool + lds32(tab + (uint32_t)offsetof(Tab, huff)), top >> 16);
    const bool is_ac = lds32(tab + (uint32_t)offsetof(Tab, is_ac)) != 0;
    return make_uint2(sizeof(Tab) == sizeof(SyncTab) ? sync_entry(c, is_ac) : value_entry(c, is_ac), c);
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
    const uint32_t next = (i0 < len && len - i0 > 16) ? __ldg(in + i0 + 16) : 0u;
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
    wait_for_previous();
    if (blockIdx.x >= w.us_tiles.total) {
        const uint32_t k = blockIdx.x - w.us_tiles.total;
        const uint2 ids = w.table_pairs[k / kTableParts];
        build_table(reinterpret_cast<CodeTables*>(w.codes)[k / kTableParts], w.huff, ids.x, ids.y, k % kTableParts, threadIdx.x, kUnstuffThreads);
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
    wait_for_previous();
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
        if (tid == 0) { w.us_len[o] = min(total, kMaxStream); w.seg_found[o] = rbase + (tot >> 16) + 1; }
    }
}

void launch_unstuff(const JpegWave& w, cudaStream_t s) {
    if (!w.n) return;
    launch_after(k_unstuff_count, w.us_tiles.total + w.n_pairs * kTableParts, kUnstuffThreads, 0, s, w);
    launch_after(k_unstuff_write, w.us_tiles.total, kUnstuffThreads, 0, s, w);
}

// ---------------------------------------------------------------------------------------------------------------
// K1  Huffman entropy decode of images without restart markers, in two kernels.
//
// The only decoder state between two blocks is (bit position p, block index c inside the MCU): the tables and the meaning
// of the next symbol follow from it.  The stream is cut into cells of CELL (1024 or 512) bits; what the second kernel needs
// is, for every cell, the state at the first block that starts in it and that block's index in the image.
//
//  k_huff_guess  Huffman streams re-synchronise: a decoder started at a wrong place soon stands where the right one does.
//     What takes long on subsampled images is the phase c, because only code lengths tell the tables apart.  Measured on
//     4:2:0 photographs (cells of 1024 bits): one decoder started 256 bits before a cell as if in block 0 of an MCU is
//     right at the cell for 25 to 58 % of the cells, but of the decoders started there in each of the MCU's blocks one is
//     right for 96 to 99 %.  So all of them run: one thread per cell and block of the MCU goes through the lead, states
//     that have met are dropped, and the distinct ones (two to four of six) decode the cell, packed into as few warps as
//     they fill.  Nothing but code lengths matters here, so symbols are looked up several at a time and no value is ever
//     extracted.  Every cell's work is independent of every other's.
//  k_huff_chain  links them: a cell's entry state is the exit state of the cell before it, and its own exit is what
//     k_huff_guess found for that entry.  One CTA per image; a thread owns a run of consecutive cells, follows the
//     candidates through it, then compares what its left neighbour hands over with what it assumed, and so on until
//     nothing changes; states nobody guessed are then decoded, all at once, and it goes on.  Chains of wrong phases are 5
//     to 15 cells long: resolving them by decoding, with one guess per cell, took 12 rounds of a cell each for a photo of
//     2.7 Mbit (276 us in a cluster of eight CTAs; 19 + 34 us for these two kernels now).
//  k_huff_write  one thread per cell decodes the blocks that start in it, values included, collects a block in shared
//     memory and writes it out whole: DC difference and class to diff[], the rows the class covers to coef[].
//
//  What bounds all three is the way of one lane: a chain of dependent instructions per symbol, with three to five warps per
//  scheduler to hide it, or one where there is little work.  So a step is few instructions (SyncTab, ValueTab), none of them a
//  jump (SyncLane::run_to, decode_blocks), and what it needs next is on its way before (Cursor, SyncLane::nx).  Before / after
//  these three, us: values 43 / 21 (one thumbnail), 51 / 28 (one photo), 1 340 / 890 (256 files of 5 Mbit); candidates 19 / 15
//  (thumbnail), 789 / 624 (256 files), 58 / 51 (8 files of 4:4:4, which now take twice the lead and 60, see kLead); restart segments
//  732 / 530 (512 files of 0.4 Mbit).
// ---------------------------------------------------------------------------------------------------------------
namespace {

// Where a decoder stands inside the MCU: the DC table of the current block as a shared-memory address (the AC table follows
// it), the tables' `off`, and the entry of the block after it.  One read per block instead of arithmetic on indices.
struct alignas(16) McuBlock { uint32_t dc; int32_t dc_off, ac_off; uint32_t next; };
__device__ __forceinline__ McuBlock lds_mcu(uint32_t a) {
    McuBlock v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.dc), "=r"(v.dc_off), "=r"(v.ac_off), "=r"(v.next) : "r"(a));
    return v;
}
// index inside the MCU of the block whose entry names `next`
__device__ __forceinline__ uint32_t mcu_index(uint32_t mcu0, uint32_t next, uint32_t bpm) {
    const uint32_t n = (next - mcu0) / (uint32_t)sizeof(McuBlock);
    return (n ? n : bpm) - 1u;
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
        const Tab* const tabs = reinterpret_cast<const Tab*>(w.codes + (size_t)(slot == 0 ? p0 : slot == slot1 ? p1 : p2) * kCodeTablesBytes + which);
        mcu[tid] = McuBlock{at, tabs[0].off, tabs[1].off, smem_addr(&mcu[(uint32_t)tid + 1 == d.bpm ? 0 : tid + 1])};
    }
}

// Streams in shared memory: a lane's window is two words (w0 holds its current bit) and the one behind them, which is on its way
// while they are used; `at` is the address of the first.  base: the address bit 0 of the stream would have.  step: the window
// moves on by a word where `crossed` is not zero; predicated by hand, because some lane of a warp crosses in nearly every step.
struct SharedSource {
    struct Cursor { uint32_t at, w2; };
    uint32_t base;
    __device__ __forceinline__ Cursor start(uint32_t& w0, uint32_t& w1, uint32_t p) const {
        const uint32_t at = base + ((p >> 3) & ~3u);
        w0 = lds32(at); w1 = lds32(at + 4);
        return Cursor{at, lds32(at + 8)};
    }
    __device__ __forceinline__ void step(uint32_t& w0, uint32_t& w1, Cursor& cur, uint32_t crossed) const {
        asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %4, 0;\n @q mov.u32 %0, %1;\n @q mov.u32 %1, %2;\n @q ld.shared.u32 %2, [%3+12];\n @q add.u32 %3, %3, 4;\n}"
                     : "+r"(w0), "+r"(w1), "+r"(cur.w2), "+r"(cur.at) : "r"(crossed));
    }
};
// ... and in global memory; `at` is the index of the first word
struct GlobalSource {
    struct Cursor { uint32_t at, w2; };
    const uint32_t* words;
    uint32_t n;
    __device__ __forceinline__ uint32_t word(uint32_t i) const { return i < n ? load_global(words + i) : 0u; }
    __device__ __forceinline__ Cursor start(uint32_t& w0, uint32_t& w1, uint32_t p) const {
        w0 = word(p >> 5); w1 = word((p >> 5) + 1);
        return Cursor{p >> 5, word((p >> 5) + 2)};
    }
    __device__ __forceinline__ void step(uint32_t& w0, uint32_t& w1, Cursor& cur, uint32_t crossed) const {
        if (crossed) { w0 = w1; w1 = cur.w2; cur.w2 = word(++cur.at + 2); }
    }
};

// A lane of a synchronising decoder.
template <class Source>
struct SyncLane {
    uint32_t base, at;   // a word boundary of the stream; the lane's place (see SyncTab), its bit position counted from there
    uint32_t nb;         // blocks ended since nb was last set to zero
    uint32_t w0, w1, tab;
    typename Source::Cursor cur;
    int32_t off;
    uint32_t ac;         // AC table of the current block
    int32_t ac_off;
    McuBlock nx;         // of the block after it
    // at a block start, or (`inside`) as if the DC term of the block had been passed
    __device__ __forceinline__ void start(const Source& src, uint32_t mcu0, uint32_t bit, bool inside, uint32_t c) {
        base = bit & ~31u; at = (bit & 31u) | (inside ? 1u << 16 : 0u); nb = 0;
        cur = src.start(w0, w1, bit);
        const McuBlock mb = lds_mcu(mcu0 + c * (uint32_t)sizeof(McuBlock));
        ac = mb.dc + (uint32_t)sizeof(SyncTab);
        ac_off = mb.ac_off;
        tab = inside ? ac : mb.dc;
        off = inside ? ac_off : mb.dc_off;
        nx = lds_mcu(mb.next);
    }
    __device__ __forceinline__ uint32_t pos() const { return base + (at & kPosMask); }
    __device__ __forceinline__ uint32_t index(uint32_t mcu0, uint32_t bpm) const {  // of the current block, inside the MCU
        const uint32_t k = mcu_index(mcu0, nx.next, bpm);
        return (k ? k : bpm) - 1u;
    }
    // One look-up: an entry of 0 (a lane that is not `live`, a rare code) changes nothing.
    __device__ __forceinline__ void apply(uint32_t e, bool& live, uint32_t stop_at, const Source& src) {
        const uint32_t was = at;
        at = was + __byte_perm(e, 0u, 0x4140);                        // all symbols
        if (at & (64u << 16)) at = was + __byte_perm(e, 0u, 0x4342);  // slot 64: the first alone
        src.step(w0, w1, cur, (was ^ at) & 32u);
        if (e) { tab = ac; off = ac_off; }
        const uint32_t end = at & kEndMask;
        // the next block, whose tables are here already
        asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %9, 0;\n @q mov.u32 %0, %5;\n @q mov.u32 %1, %6;\n @q add.u32 %2, %5, %10;\n @q mov.u32 %3, %7;\n"
                     " @q add.u32 %4, %4, 1;\n @q ld.shared.v4.u32 {%5,%6,%7,%8}, [%8];\n}"
                     : "+r"(tab), "+r"(off), "+r"(ac), "+r"(ac_off), "+r"(nb), "+r"(nx.dc), "+r"(nx.dc_off), "+r"(nx.ac_off), "+r"(nx.next)
                     : "r"(end), "n"((int)sizeof(SyncTab)));
        if (end) { at &= kPosMask; live = at < stop_at; }
    }
    // Lanes with `live` decode to the first block start at a position of at least `stop`.  Called by whole warps: the loop has
    // one exit, taken by all lanes together, and no other jump out of it -- with returns from inside, the lanes of a warp
    // never met again after their first different turn and went on alone.  The steps themselves are free of branches: a lane
    // waits for every instruction of its chain, and jumps were a third of the chain.
    __device__ __forceinline__ void run_to(bool live, uint32_t stop, const Source& src, const HuffTable* pool) {
        const uint32_t stop_at = stop > base ? stop - base : 0u;
        while (__any_sync(0xFFFFFFFFu, live)) {
            uint32_t e = 0;
#pragma unroll
            for (int step = 0; step < 4; ++step) {
                e = entry_at<SyncTab>(tab, off, __funnelshift_l(w1, w0, at));
                apply(live ? e : 0u, live, stop_at, src);
            }
            if (live && e == 0) apply(rare_entry<SyncTab>(tab, __funnelshift_l(w1, w0, at), pool).x, live, stop_at, src);
        }
    }
};

// Streams staged in shared memory: consecutive cells.  A block may run 1984 bits (64 symbols of 31 bits) into what follows the
// last cell, and the padding of a stream covers that: kRowsBehind, kRowsPadded.  (Cells of 1024 bits start in the same bank;
// padding them apart costs more instructions per symbol than the conflicts of the few lanes that load in one step.)
template <int CELL>
struct Staged {
    static constexpr int kPitch = CELL / 8, kRowsBehind = 1984 / CELL + 2, kRowsPadded = 2048 / CELL;
    // cells [row0, row0 + rows) of the stream `us`
    static __device__ __forceinline__ void copy(unsigned char* stage, const uint8_t* us, uint32_t row0, int rows, int tid, int nthreads) {
        const uint8_t* src = us + (size_t)row0 * kPitch;
        const uint32_t dst = smem_addr(stage);
        for (int i = tid; i < rows * (kPitch / 16); i += nthreads) copy16(dst + i * 16, src + i * 16);
        copy_commit();
    }
};
static_assert(kStreamPad >= (2048 + 1024) / 8 + 16, "rows behind the end of a stream are copied");
static_assert((1ull << 32) - kMaxStream * 8ull > 2ull * kDecodeThreadsMany * kCellBits + 4096, "positions behind the end of a stream do not wrap");

// A state at or behind the first bit of a cell, relative to it: bits 0-11 distance of the block start (less than 2048: a
// block has 64 symbols of 31 bits at most), 12-14 its block c.
constexpr uint32_t kStNone = 0xFFFFu, kStDropped = 0xFFFEu;  // the stream ends before; no candidate
__device__ __forceinline__ uint32_t pack_state(uint32_t p, uint32_t cell_bit, uint32_t c, uint32_t total) { return p > total ? kStNone : (p - cell_bit) | c << 12; }

// Where cell k of an image stands in w.cells and w.cand.  A thread of the linking kernel walks `run` consecutive cells.  Where
// runs are long (`mixed`, see JpegWave), the cells that all threads read in the same step are neighbours instead: in order, a load
// of a warp touched 32 lines, and the loads of a step queued for 2 900 cycles (8 images of 4:4:4, up to 17 cells a thread: 66 us
// for the kernel, 50 like this, and 39 with the longer lead on top).
struct CellOrder {
    uint32_t run, threads;
    bool mixed;
    __device__ __forceinline__ CellOrder(uint32_t ncell, uint32_t threads, bool mixed) : run((ncell + threads - 1) >> (threads == 256 ? 8 : 10)), threads(threads), mixed(mixed) {}
    __device__ __forceinline__ uint32_t at(uint32_t k) const {
        if (!mixed) return k;
        const uint32_t t = k / run;
        return (k - t * run) * threads + t;
    }
    // pieces of two candidates: in order all of a cell's together, else one of each cell together
    static constexpr uint32_t kPieces = kCandidates / 2;
    __device__ __forceinline__ uint32_t piece_step() const { return mixed ? run * threads : 1u; }  // from a cell's piece to its next one
    __device__ __forceinline__ uint32_t piece(uint32_t k, uint32_t h) const { return mixed ? h * piece_step() + at(k) : k * kPieces + h; }
};

// Bits before a cell from which its candidates are decoded.  512 leave a third of the open states that 256 leave; that costs the
// candidates 3 us and saves a long stream's linking more (one photo of 5 234 cells: 16.3 + 41.3 us with 256, 19.1 + 33.9 with 512;
// 8 images of 4:4:4: 51 + 50 and 60 + 39; a thumbnail of 312 cells has few open states anyway).
constexpr uint32_t kLead = 256, kLeadMixed = 512;
constexpr int kGuessThreads = (int)kGuessLanes;

}  // namespace

// A CTA takes guess_spans() spans of w.guess_span cells, a thread per span and block of the MCU.  Decoders that meet are one
// from then on, so in a span of several cells the lead is run once and fewer decoders are left from cell to cell; with few
// images a span is one cell, because then the length of a thread's way is what counts.
template <int CELL, bool MIXED>
__global__ void __launch_bounds__(kGuessThreads) k_huff_guess(JpegWave w) {
    extern __shared__ __align__(16) unsigned char guess_smem[];
    __shared__ McuBlock mcu[6];
    __shared__ uint16_t s_state[kGuessThreads], s_list[kGuessThreads];
    __shared__ uint32_t s_warp[kGuessThreads / 32];
    const uint32_t o = owner_of(w.guess_ctas, blockIdx.x);
    const uint32_t img = w.spec_list[o];
    const JpegDesc& d = w.descs[img];
    const uint32_t bpm = d.bpm;
    wait_for_previous();
    const uint32_t span = w.guess_span, nspans = guess_spans(bpm, span), cell0 = (blockIdx.x - __ldg(w.guess_ctas.first + o)) * nspans * span;
    const uint32_t total = w.us_len[img] * 8u, ncell = (total + CELL - 1) / CELL;
    if (cell0 >= ncell) return;
    unsigned char* const tab0 = guess_smem;
    unsigned char* const stage = tab0 + w.max_pairs * 2 * sizeof(SyncTab);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr uint32_t lead = MIXED ? kLeadMixed : kLead;
    static_assert(lead <= (uint32_t)CELL, "the lead lies in the cell before");
    const uint32_t row0 = cell0 ? cell0 - 1 : 0, cell1 = min(cell0 + nspans * span, ncell);
    Staged<CELL>::copy(stage, w.us + d.us_off, row0, (int)(min(cell0 + nspans * span + Staged<CELL>::kRowsBehind, ncell + Staged<CELL>::kRowsPadded) - row0), tid, kGuessThreads);
    load_tables<SyncTab>(w, d, mcu, tab0, (uint32_t)offsetof(CodeTables, sync), tid, kGuessThreads);
    copy_commit();
    const CellOrder order(ncell, 1024, MIXED);
    uint2* const cand = reinterpret_cast<uint2*>(w.cand + (size_t)d.cell_off * CellOrder::kPieces);
    for (uint32_t i = cell0 * (kCandidates / 2) + tid; i < cell1 * (kCandidates / 2); i += kGuessThreads)
        reinterpret_cast<uint4*>(cand)[order.mixed ? order.piece(i / CellOrder::kPieces, i % CellOrder::kPieces) : i] = make_uint4(kStDropped, 0, kStDropped, 0);
    copy_wait<0>();
    __syncthreads();
    const uint32_t mcu0 = smem_addr(&mcu[0]);
    const SharedSource source{smem_addr(stage) - row0 * (uint32_t)Staged<CELL>::kPitch};

    // ---- the lead: from its first bit on, as if inside each of the MCU's blocks
    const uint32_t mine = cell0 + (uint32_t)tid / bpm * span, myh = (uint32_t)tid % bpm;  // first cell of this thread's span
    const bool live = (uint32_t)tid < nspans * bpm && mine < ncell;
    uint32_t k = live ? mine : cell0;
    SyncLane<SharedSource> L{};
    L.start(source, mcu0, k ? k * CELL - lead : 0u, k != 0u, live && k ? myh : 0u);
    L.run_to(live && k, k * CELL, source, w.huff);
    uint32_t decodes = 0;
    s_state[tid] = (uint16_t)(live ? pack_state(L.pos(), k * CELL, L.index(mcu0, bpm), total) : kStNone);
    for (uint32_t step = 0; step < span; ++step) {
        __syncthreads();
        // ---- the distinct states, in as few warps as they fill
        const uint32_t state = s_state[tid];
        bool keep = state < kStDropped && mine + step < ncell;
        for (uint32_t i = 1; keep && i <= myh; ++i) keep = s_state[tid - i] != state;
        const uint32_t kept = __ballot_sync(0xFFFFFFFFu, keep);
        if (lane == 0) s_warp[warp] = __popc(kept);
        __syncthreads();
        if (!keep) s_state[tid] = (uint16_t)kStDropped;
        uint32_t before = 0, all = 0;
#pragma unroll
        for (int i = 0; i < kGuessThreads / 32; ++i) { const uint32_t n = s_warp[i]; if (i < warp) before += n; all += n; }
        decodes += all;
        if (keep) s_list[before + __popc(kept & ((1u << lane) - 1u))] = (uint16_t)tid;
        __syncthreads();
        // ---- through their cell
        if ((uint32_t)warp * 32u < all) {
            const bool on = (uint32_t)tid < all;
            const uint32_t t = s_list[on ? tid : warp * 32], entry = s_state[t];
            k = cell0 + t / bpm * span + step;
            const uint32_t bound = (k + 1) * CELL, p = k * CELL + (entry & 0xFFFu);
            L.start(source, mcu0, p, false, entry >> 12);
            L.run_to(on && p < bound, min(bound, total + 1), source, w.huff);
            __syncwarp();
            if (on) {
                const uint32_t exit = pack_state(L.pos(), bound, L.index(mcu0, bpm), total);
                if (L.pos() > total) --L.nb;  // the block that ended here is not whole
                const uint32_t h = t % bpm;
                cand[order.mixed ? (size_t)order.piece(k, h / 2) * 2 + (h & 1u) : (size_t)k * kCandidates + h] = make_uint2(entry | exit << 16, L.nb);
                s_state[t] = (uint16_t)exit;
            }
        }
    }
    if (tid == 0) atomicAdd(w.spec_stats + 2, (unsigned long long)decodes);
}

namespace {

template <int T>
struct ChainMisc {
    uint32_t exit[T];      // state each thread hands to its right neighbour
    McuBlock mcu[6];
    uint32_t warp[32];
};
static_assert(sizeof(ChainMisc<256>) % 16 == 0, "tables follow in shared memory");

}  // namespace

template <int T, int CELL, bool MIXED>
__global__ void __launch_bounds__(T) k_huff_chain(JpegWave w) {
    extern __shared__ __align__(16) unsigned char chain_smem[];
    ChainMisc<T>& sh = *reinterpret_cast<ChainMisc<T>*>(chain_smem);
    unsigned char* const tab0 = chain_smem + sizeof(ChainMisc<T>);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t img = w.spec_list[blockIdx.x];
    const JpegDesc& d = w.descs[img];
    wait_for_previous();
    load_tables<SyncTab>(w, d, sh.mcu, tab0, (uint32_t)offsetof(CodeTables, sync), tid, T);
    copy_commit();
    const uint32_t us_len = w.us_len[img], total = us_len * 8u;
    const uint32_t ncell = (total + CELL - 1) / CELL;
    const GlobalSource source{from_previous(reinterpret_cast<const uint32_t*>(w.us + d.us_off)), (us_len + 3) / 4 + 2};
    const CellOrder order(ncell, T, MIXED);
    const uint32_t run = order.run, kbeg = min(tid * run, ncell), kend = min(kbeg + run, ncell);
    // of this thread's cell k: [(k - kbeg) * step]
    const uint32_t step = order.mixed ? T : 1, cand_step = order.mixed ? T : CellOrder::kPieces, piece = order.piece_step();
    uint2* const recs = w.cells + d.cell_off + 1 + tid * (order.mixed ? 1 : run);  // while linking: block start, state << 12 | blocks that start in the cell
    const uint4* const cand = from_previous(w.cand) + (size_t)d.cell_off * CellOrder::kPieces + tid * (order.mixed ? 1 : run * CellOrder::kPieces);
    const bool active = kbeg < kend;
    const uint32_t mcu0 = smem_addr(&sh.mcu[0]);
    uint32_t found = 0;  // blocks that start in this thread's cells
    uint32_t exit = kStNone;
    copy_wait<0>();
    __syncthreads();

    // Follows the candidates from `state` at cell `k` on.  Walking again (`redo`), it stops at a cell whose recorded state it
    // meets, unless something behind that cell is still open.  A state that is no candidate of its cell is left open
    // (open_at, open_state): the cells from there on keep what they have, on the first walk a chain of their own.
    uint32_t open_at = ~0u, open_state = 0, last_open = 0;  // last_open: no cell from here on is open
    auto follow = [&](bool live, uint32_t k, uint32_t state, bool redo) {
        if (live) open_at = ~0u;
        const bool on = live && k < kend;
        uint32_t still_open = 0;
        for (const uint32_t first = k; on; ++k) {
            const uint32_t cell_bit = k * CELL;
            uint32_t next = kStNone, n = 0;
            uint2 had = make_uint2(0, 0);
            if (redo) {
                had = recs[(k - kbeg) * step];
                if (k != first && k >= last_open && (had.y >> 12) == state) break;  // met
            }
            if (state != kStNone) {
                if ((state & 0xFFFu) >= (uint32_t)CELL) next = state - CELL;  // no block starts in this cell
                else {
                    const uint4* const c = cand + (k - kbeg) * cand_step;
                    const uint4 a = load_global(c), b = load_global(c + piece), e = load_global(c + 2 * piece);
                    bool known = false;
                    auto look = [&](uint32_t x, uint32_t y) { if ((x & 0xFFFFu) == state) { next = x >> 16; n = y; known = true; } };
                    look(a.x, a.y); look(a.z, a.w); look(b.x, b.y); look(b.z, b.w); look(e.x, e.y); look(e.z, e.w);
                    if (!known) {
                        if (open_at == ~0u) { open_at = k; open_state = state; }
                        still_open = k + 1;
                        if (redo) { still_open = max(still_open, last_open); break; }
                        state = a.x & 0xFFFFu;
                        if (state == kStDropped) state = kStNone;
                        else { next = a.x >> 16; n = a.y; }
                    }
                }
            }
            recs[(k - kbeg) * step] = make_uint2(state == kStNone ? kNoState : cell_bit + (state & 0xFFFu), state << 12 | n);
            found += n - (had.y & 0xFFFu);
            state = next;
            if (k + 1 == kend) { exit = state; break; }
        }
        if (on) last_open = still_open;
    };

    uint32_t entry = 0;  // thread 0: bit 0, block 0
    if (active && tid) {
        entry = load_global(&cand->x) & 0xFFFFu;
        if (entry == kStDropped) entry = kStNone;
    }
    follow(active, kbeg, entry, false);
    sh.exit[tid] = exit;
    uint32_t decodes = active ? kend - kbeg : 0u, rounds = 1, round = 0;  // decodes: once each for the values, and those below
    __syncthreads();
    // Look-ups until nothing changes any more; then what is open is decoded, one cell per thread; and again.  Opened cells have
    // their turn in every eighth round in any case: of eight rounds, one settles the first thread that is not final yet or
    // its next open cell, which bounds the rounds (a photo takes 10 to 30, one to three of them decoding).
    const uint64_t limit = 8ull * (ncell + T) + 8;
    for (; round <= limit; ++round) {
        const uint32_t prev = active && tid ? sh.exit[tid - 1] : entry;
        const bool need = prev != entry, any_need = __syncthreads_or(need);
        const bool decode = open_at != ~0u;
        bool any_decode = false;
        if (!any_need || (round & 7u) == 7u) any_decode = __syncthreads_or(decode);
        if (!any_need && !any_decode) break;
        if (!any_decode) {
            if (need) entry = prev;
            follow(need, kbeg, entry, true);
        } else {
            if (__any_sync(0xFFFFFFFFu, decode)) {
                const uint32_t k = decode ? open_at : 0, bound = (k + 1) * CELL, p = k * CELL + (decode ? open_state & 0xFFFu : 0u);
                SyncLane<GlobalSource> L;
                L.start(source, mcu0, p, false, decode ? open_state >> 12 : 0u);
                L.run_to(decode, min(bound, total + 1), source, w.huff);
                __syncwarp();
                if (decode) {
                    ++decodes;
                    const uint32_t n = L.nb - (L.pos() > total ? 1u : 0u), next = pack_state(L.pos(), bound, L.index(mcu0, d.bpm), total);
                    found += n - (recs[(k - kbeg) * step].y & 0xFFFu);
                    recs[(k - kbeg) * step] = make_uint2(p, open_state << 12 | n);
                    if (k + 1 == kend) { exit = next; open_at = ~0u; last_open = 0; }
                    else follow(true, k + 1, next, true);
                }
            }
        }
        sh.exit[tid] = exit;
        ++rounds;
        __syncthreads();
    }
    // index of the first block of every cell
    uint32_t inc = found;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o); if (lane >= o) inc += t; }
    if (lane == 31) sh.warp[warp] = inc;
    decodes = __reduce_add_sync(0xFFFFFFFFu, decodes);
    if (lane == 0) atomicAdd(w.spec_stats + 2, (unsigned long long)decodes);
    __syncthreads();
    uint32_t base = inc - found;
#pragma unroll
    for (int i = 0; i < T / 32; ++i) if (i < warp) base += sh.warp[i];
#pragma unroll 4
    for (uint32_t i = 0; i < kend - kbeg; ++i) { const uint32_t n = recs[i * step].y & 0xFFFu; recs[i * step].y = base; base += n; }
    if (tid == T - 1) {
        w.cells[d.cell_off] = make_uint2(kNoState, base);
        uint32_t err = 0;
        if (base < d.nblocks) err |= kStTruncated;
        if (round > limit) err |= kStSyncLimit;
        if (err) atomicOr(w.status + d.item, err);
        atomicAdd(w.spec_stats, (unsigned long long)ncell);
        atomicAdd(w.spec_stats + 1, (unsigned long long)rounds);
    }
}

// ---- blocks with their values --------------------------------------------------------------------------------------
namespace {

constexpr uint32_t kBlankBlock = (uint32_t)kClsDc << 16;  // in info[]: a block the stream does not hold
constexpr uint32_t kNotDc = 1u, kNot2x2 = 2u, kNot4x4 = 4u;

// Zig-zag position -> byte offset of the coefficient in a lane's block buffer (row r of the lane's block sits at
// r * T * 16: rows of neighbouring lanes are neighbours, so whole-row accesses are conflict free) << 16 | class flags.
template <int T>
__device__ __forceinline__ uint32_t place_of(uint32_t zz) {
    static_assert(8 * T * 16 <= 65536, "offsets are 16-bit numbers");
    const uint32_t nat = kNatural[zz], r = nat >> 3, c = nat & 7u;
    return (r * (T * 16) + c * 2) << 16 | (zz ? kNotDc : 0u) | (r > 1 || c > 1 ? kNot2x2 : 0u) | (r > 3 || c > 3 ? kNot4x4 : 0u);
}

template <int T>
struct ValueMisc {
    uint4 block[8 * T];    // the lanes' current blocks
    uint32_t place[64];
    McuBlock mcu[6];
};

// Shared memory of the value decoder: [ValueMisc | ... | tables].
template <int T>
__device__ __forceinline__ void value_setup(ValueMisc<T>& sh) {
    const int tid = threadIdx.x;
    if (tid < 64) sh.place[tid] = place_of<T>(tid);
#pragma unroll
    for (int r = 0; r < 8; ++r) sh.block[r * T + tid] = make_uint4(0, 0, 0, 0);
}
// ... and its tables; the caller waits for the copies and the barrier.
template <int T>
__device__ __forceinline__ void value_tables(const JpegWave& w, const JpegDesc& d, ValueMisc<T>& sh, unsigned char* tab0) {
    load_tables<ValueTab>(w, d, sh.mcu, tab0, (uint32_t)offsetof(CodeTables, value), threadIdx.x, T);
    copy_commit();
}

// Decodes blocks [blk, end) of an image from bit p on.  src: the image's stream, see SharedSource.
// limit: blocks that reach beyond this bit are not whole -- decoding stops there; so it does at a block that starts at or
// behind `stop`.  ABSOLUTE: the DC predictors start at zero here (a restart segment) and info[] receives the DC terms
// themselves instead of their differences.  Returns the blocks decoded.  Called by whole warps.
//
// One code path for DC and AC symbols, the DC difference going to slot 0 of the block buffer like any coefficient: the lanes
// of a warp are at unrelated places.  For the same reason a lane whose block is complete waits until kFlushLanes lanes
// have one (or no lane has anything else to do): writing a block out takes more instructions than decoding a symbol,
// and they cost the same whether two lanes execute them or ten.  The warp looks for such lanes after every other symbol.
constexpr int kFlushLanes = 8;

template <int T, bool ABSOLUTE, class Source>
__device__ __forceinline__ uint32_t decode_blocks(const Source& src, const uint32_t p, uint32_t blk, const uint32_t end, const uint32_t limit, const uint32_t stop,
                                                  uint32_t c, const JpegDesc& d, ValueMisc<T>& sh, const HuffTable* pool, int16_t* __restrict__ coef,
                                                  uint32_t* __restrict__ info, uint32_t& err) {
    const uint32_t first = blk, mcu0 = smem_addr(&sh.mcu[0]);
    bool live = blk < end;
    uint32_t w0, w1;
    typename Source::Cursor cur = src.start(w0, w1, p);
    uint32_t base = p & ~31u, at = p & 31u;  // of the current block: a word boundary, the lane's place (see ValueTab)
    const uint32_t place = smem_addr(sh.place) - 4, buf = smem_addr(&sh.block[threadIdx.x]);
    McuBlock mb = lds_mcu(mcu0 + c * (uint32_t)sizeof(McuBlock));
    uint32_t tab = mb.dc, seen = 0, last = 0;  // last: the entry of the last symbol
    int32_t off = mb.dc_off;
    int32_t pred0 = 0, pred1 = 0, pred2 = 0;
    // one symbol; an entry of 0 (a lane that waits, a rare code) changes nothing
    const auto apply = [&](uint32_t e, uint32_t top) {
        const uint32_t was = at;
        at += e;
        src.step(w0, w1, cur, (was ^ at) & 32u);
        // the s extra bits (T.81 EXTEND), first moved to the top: a leading 1 means the value itself, a leading 0 the complement
        // of its magnitude
        const uint32_t n = e >> 27, bits = __funnelshift_l(0u, __funnelshift_l(top, 0u, e), n);
        const uint32_t neg = ~(uint32_t)((int32_t)bits >> 31);
        const uint32_t v = __funnelshift_r(bits, neg, n) - neg;
        const uint32_t slot = at >> 14 & 0x3FCu;  // (times four)
        const bool store = (int32_t)e < 0 && slot <= 256u;
        asm volatile("{\n .reg .pred q;\n .reg .u32 a, o;\n .reg .u16 h;\n setp.ne.u32 q, %1, 0;\n @q ld.shared.u32 a, [%2];\n cvt.u16.u32 h, %3;\n"
                     " shr.u32 o, a, 16;\n add.u32 o, o, %4;\n @q st.shared.u16 [o], h;\n @q or.b32 %0, %0, a;\n}"
                     : "+r"(seen) : "r"((uint32_t)store), "r"(place + slot), "r"(v), "r"(buf) : "memory");
        if (e) { tab = mb.dc + (uint32_t)sizeof(ValueTab); off = mb.ac_off; last = e; }
    };
    for (;;) {
        const uint32_t alive = __ballot_sync(0xFFFFFFFFu, live);
        if (!alive) break;  // one exit for the whole warp, see SyncLane::run_to
        uint32_t e = 0;
#pragma unroll
        for (int step = 0; step < 2; ++step) {
            const uint32_t top = __funnelshift_l(w1, w0, at);
            e = entry_at<ValueTab>(tab, off, top);
            apply(live && !(at & kEndMask) ? e : 0u, top);
        }
        if (e == 0 && live && !(at & kEndMask)) {
            const uint32_t top = __funnelshift_l(w1, w0, at);
            const uint2 rare = rare_entry<ValueTab>(tab, top, pool);
            if (rare.y >> 31 && base + (at & kPosMask) < limit) err |= kStBadCode;
            apply(rare.x, top);
        }
        const uint32_t done = __ballot_sync(0xFFFFFFFFu, live && (at & kEndMask));
        if (__popc(done) >= kFlushLanes || done == alive) {
            if (live && (at & kEndMask)) {
                const uint32_t now = base + (at & kPosMask);
                if (now > limit) live = false;  // (what the buffer holds is of no use, and neither is the rest of the span)
                else {
                    if ((int32_t)last < 0 && (at >> 14 & 0x3FCu) > 256u) err |= kStCoefRange;
                    uint4* const b = sh.block + threadIdx.x;
                    uint4* const rows = reinterpret_cast<uint4*>(coef) + (size_t)blk * 8;
                    const uint4 zero = make_uint4(0, 0, 0, 0), q0 = b[0];
                    int32_t dc = (int16_t)(q0.x & 0xFFFFu);
                    if (ABSOLUTE) {
                        const uint32_t luma = d.hs * d.vs, k = mcu_index(mcu0, mb.next, d.bpm);
                        if (k < luma) dc = pred0 += dc;
                        else if (k == luma) dc = pred1 += dc;
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
                    live = blk < end && now < stop;
                    base = now & ~31u; at = now & 31u;
                    seen = 0;
                    mb = lds_mcu(mb.next);
                    tab = mb.dc;
                    off = mb.dc_off;
                }
            }
        }
    }
    return blk - first;
}

}  // namespace

// ---- restart-free images: one thread per cell -----------------------------------------------------------------------
// The CTA's T cells are consecutive: their stream is staged in shared memory.
template <int T, int CELL>
__global__ void __launch_bounds__(T) k_huff_write(JpegWave w) {
    extern __shared__ __align__(16) unsigned char write_smem[];
    ValueMisc<T>& sh = *reinterpret_cast<ValueMisc<T>*>(write_smem);
    unsigned char* const stage = write_smem + sizeof(ValueMisc<T>);
    unsigned char* const tab0 = stage + (T + Staged<CELL>::kRowsBehind) * Staged<CELL>::kPitch;
    const uint32_t o = owner_of(w.write_ctas, blockIdx.x);
    const uint32_t img = w.spec_list[o];
    const JpegDesc& d = w.descs[img];
    const uint32_t cell0 = (blockIdx.x - __ldg(w.write_ctas.first + o)) * T;
    const int tid = threadIdx.x;
    value_setup<T>(sh);
    wait_for_previous();
    const uint32_t total = w.us_len[img] * 8u;
    const uint32_t ncell = (total + CELL - 1) / CELL;
    if (cell0 >= ncell) return;
    // (no further than the stream and its padding reach)
    Staged<CELL>::copy(stage, w.us + d.us_off, cell0, (int)min((uint32_t)(T + Staged<CELL>::kRowsBehind), ncell - cell0 + Staged<CELL>::kRowsPadded), tid, T);
    value_tables<T>(w, d, sh, tab0);
    const uint32_t k = cell0 + tid;
    const CellOrder order(ncell, w.chain_threads, w.mixed);
    const uint2* recs = w.cells + d.cell_off;
    uint2 a = make_uint2(0, 0);
    uint32_t b1 = 0;
    if (k < ncell) {
        a = recs[1 + order.at(k)];
        b1 = min(recs[k + 1 < ncell ? 1 + order.at(k + 1) : 0].y, d.nblocks);
    }
    copy_wait<0>();
    __syncthreads();
    uint32_t err = 0;
    const SharedSource source{smem_addr(stage) - cell0 * (uint32_t)Staged<CELL>::kPitch};
    const uint32_t p0 = a.y < b1 ? a.x : cell0 * CELL;
    decode_blocks<T, false>(source, p0, a.y, b1, total, (cell0 + T) * CELL, a.y % d.bpm, d, sh, w.huff,
                                        w.coef + d.block_off * 64, w.diff + d.block_off, err);
    if (err) atomicOr(w.status + d.item, err);
}

// ---- restart-interval images: one thread per segment -----------------------------------------------------------------
// A segment's first MCU and the zero DC predictors are known, so one pass does it.  The segments of a CTA are consecutive
// in one image; the stream under them is staged when it fits (it does for intervals of a few MCUs), else read in place.
template <int T> constexpr uint32_t kRestartStage = T * 128;

template <int T>
__global__ void __launch_bounds__(T) k_huff_restart(JpegWave w) {
    extern __shared__ __align__(16) unsigned char restart_smem[];
    ValueMisc<T>& sh = *reinterpret_cast<ValueMisc<T>*>(restart_smem);
    unsigned char* const stage = restart_smem + sizeof(ValueMisc<T>);
    unsigned char* const tab0 = stage + kRestartStage<T>;
    const uint32_t o = owner_of(w.restart_ctas, blockIdx.x);
    const uint32_t img = w.restart_list[o];
    const JpegDesc& d = w.descs[img];
    const uint32_t k0 = (blockIdx.x - __ldg(w.restart_ctas.first + o)) * T;
    const int tid = threadIdx.x;
    value_setup<T>(sh);
    wait_for_previous();
    const uint32_t found = w.seg_found[img], us_len = w.us_len[img], k = k0 + tid;
    if (k0 == 0 && tid == 0 && found != d.nseg) atomicOr(w.status + d.item, kStBadMarker);
    const uint32_t* seg = w.seg_start + d.seg_off;
    const uint32_t have = min(found, d.nseg);  // entries of seg[] that exist
    const uint32_t mcus = d.mcux * d.mcuy;
    const uint32_t m0 = min(k * d.restart, mcus), m1 = min(m0 + d.restart, mcus);
    const uint32_t blk0 = m0 * d.bpm, blk1 = m1 * d.bpm;
    uint32_t* info = w.info + d.block_off;
    // blocks that a damaged file lacks are flat mid-gray, not what an earlier wave left in info[] and coef[]
    const auto blank = [&](uint32_t from) { for (uint32_t b = from; b < blk1; ++b) info[b] = kBlankBlock; };
    if (k0 >= have) { blank(blk0); return; }
    // the CTA's piece of the stream: from the 16-byte piece its first segment starts in to its end plus what a block that
    // is not whole may run over
    const auto begin = [&](uint32_t i) { return i < have ? min(seg[i], us_len) : us_len; };  // of a segment (us_len: see kMaxStream)
    const uint32_t lo = begin(k0) & ~15u, hi = begin(k0 + T) + 272u;
    const bool staged = hi - lo <= kRestartStage<T>;
    const uint8_t* us = w.us + d.us_off;
    if (staged) {
        const uint32_t dst = smem_addr(stage);
        for (uint32_t i = tid; i * 16 < hi - lo; i += T) copy16(dst + i * 16, us + lo + (size_t)i * 16);
        copy_commit();
    }
    value_tables<T>(w, d, sh, tab0);
    copy_wait<0>();
    __syncthreads();
    const bool mine = k < have;
    const uint32_t b0 = mine ? begin(k) : lo, b1 = begin(k + 1);
    const uint32_t end = mine ? blk1 : blk0;
    int16_t* coef = w.coef + d.block_off * 64;
    uint32_t err = 0, n;
    if (staged) {
        n = decode_blocks<T, true>(SharedSource{smem_addr(stage) - lo}, b0 * 8u, blk0, end, b1 * 8u, b1 * 8u, 0u, d, sh, w.huff, coef, info, err);
    } else {
        const GlobalSource source{from_previous(reinterpret_cast<const uint32_t*>(us)), (us_len + 3) / 4 + 2};
        n = decode_blocks<T, true>(source, b0 * 8u, blk0, end, b1 * 8u, b1 * 8u, 0u, d, sh, w.huff, coef, info, err);
    }
    if (n < end - blk0) err |= kStTruncated;
    if (n < blk1 - blk0) blank(blk0 + n);
    if (err) atomicOr(w.status + d.item, err);
}

// ---------------------------------------------------------------------------------------------------------------
// K1b  DC prediction of restart-free images: diff[] holds what info[] will hold, with DC differences, in scan order; the
//      predictor runs over the blocks of a component.  Kept out of the bit-serial kernels on purpose: there it would cost every symbol of the
//      synchronising pass a value extraction, here it is a prefix sum over four bytes per block.
//      A cluster of CTAs per image, each with an equal run of its MCUs: a CTA adds up its run, the cluster exchanges the
//      sums, and the CTA writes its run -- from registers where a thread has no more than four MCUs.  What bounds it is the
//      latency of its few dependent loads, so the blocks are fetched before it is known how many the stream holds.  (One CTA
//      per 8192 MCUs, which read again what lay before its range: 16 us for one photo, 43 for 8 images of 4:4:4 up to 4096
//      pixels.)
// ---------------------------------------------------------------------------------------------------------------
namespace {

constexpr int kDcThreads = 512;
struct Dc3 { int32_t a, b, c; };
__device__ __forceinline__ Dc3 operator+(Dc3 x, Dc3 y) { return {x.a + y.a, x.b + y.b, x.c + y.c}; }

// four MCUs per thread: BPM 16-byte pieces
template <int BPM>
__device__ __forceinline__ void load_mcus(const uint32_t* diff, uint32_t m4, uint32_t nblocks, uint32_t (&v)[4 * BPM]) {
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
}
// their differences; blocks from `have` on, which the stream does not hold, count as nothing
template <int BPM>
__device__ __forceinline__ Dc3 sum_mcus(uint32_t m4, uint32_t have, uint32_t (&v)[4 * BPM]) {
    const uint32_t b0 = m4 * 4 * BPM;
    if (b0 + 4 * BPM > have) {
#pragma unroll
        for (int i = 0; i < 4 * BPM; ++i) if (b0 + i >= have) v[i] = 0;
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

struct DcSmem { Dc3 warp[kDcThreads / 32], total, carry; };

// blocks: how many of the image's blocks the stream holds (called once the first loads are under way)
template <int BPM, class Blocks>
__device__ void dc_image(const uint32_t* diff, uint32_t* info, uint32_t nblocks, Blocks&& blocks, DcSmem& sh) {
    const auto cluster = cooperative_groups::this_cluster();
    const uint32_t rank = cluster.block_rank(), size = cluster.num_blocks();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t groups = (nblocks + 4 * BPM - 1) / (4 * BPM), run = (groups + size - 1) / size;  // of four MCUs
    const uint32_t g0 = min(rank * run, groups), g1 = min(g0 + run, groups);
    const bool once = run <= (uint32_t)kDcThreads;  // the run stays in registers
    uint32_t v[4 * BPM];
    if (g0 + tid < g1) load_mcus<BPM>(diff, g0 + tid, nblocks, v);
    const uint32_t have = blocks();
    Dc3 x{0, 0, 0};
    if (g0 + tid < g1) x = sum_mcus<BPM>(g0 + tid, have, v);
    const Dc3 first = x;
    for (uint32_t g = g0 + tid + kDcThreads; g < g1; g += kDcThreads) {
        load_mcus<BPM>(diff, g, nblocks, v);
        x = x + sum_mcus<BPM>(g, have, v);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) { x.a += __shfl_xor_sync(0xFFFFFFFFu, x.a, o); x.b += __shfl_xor_sync(0xFFFFFFFFu, x.b, o); x.c += __shfl_xor_sync(0xFFFFFFFFu, x.c, o); }
    if (lane == 0) sh.warp[warp] = x;
    __syncthreads();
    if (tid == 0) {
        Dc3 t{0, 0, 0};
#pragma unroll
        for (int i = 0; i < kDcThreads / 32; ++i) t = t + sh.warp[i];
        sh.total = t;
    }
    cluster.sync();
    if (warp == 0) {  // what the CTAs before this one add up to
        Dc3 t{0, 0, 0};
        if ((uint32_t)lane < rank) t = *cluster.map_shared_rank(&sh.total, lane);
#pragma unroll
        for (int o = 16; o; o >>= 1) { t.a += __shfl_xor_sync(0xFFFFFFFFu, t.a, o); t.b += __shfl_xor_sync(0xFFFFFFFFu, t.b, o); t.c += __shfl_xor_sync(0xFFFFFFFFu, t.c, o); }
        if (lane == 0) sh.carry = t;
    }
    cluster.barrier_arrive();  // this CTA has read the others' sums
    __syncthreads();
    Dc3 carry = sh.carry;
    // (info keeps 16 bits, so nothing is lost when a damaged stream makes the sums wrap)
    for (uint32_t g = g0; g < g1; g += kDcThreads) {
        const uint32_t m4 = g + tid;
        Dc3 mine{0, 0, 0};
        if (once) mine = first;
        else if (m4 < g1) { load_mcus<BPM>(diff, m4, nblocks, v); mine = sum_mcus<BPM>(m4, have, v); }
        Dc3 inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t ta = __shfl_up_sync(0xFFFFFFFFu, inc.a, o), tb = __shfl_up_sync(0xFFFFFFFFu, inc.b, o), tc = __shfl_up_sync(0xFFFFFFFFu, inc.c, o);
            if (lane >= o) { inc.a += ta; inc.b += tb; inc.c += tc; }
        }
        __syncthreads();
        if (lane == 31) sh.warp[warp] = inc;
        __syncthreads();
        Dc3 pre{0, 0, 0}, all{0, 0, 0};
#pragma unroll
        for (int i = 0; i < kDcThreads / 32; ++i) { const Dc3 t = sh.warp[i]; if (i < warp) pre = pre + t; all = all + t; }
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
        if (b0 + 4 * BPM <= have) {
#pragma unroll
            for (int i = 0; i < BPM; ++i) reinterpret_cast<uint4*>(info + b0)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4 * BPM; ++i) if (b0 + i < nblocks) info[b0 + i] = b0 + i < have ? v[i] : kBlankBlock;
        }
    }
    cluster.barrier_wait();  // the sums stay until every CTA has read them
}

}  // namespace

__global__ void __launch_bounds__(kDcThreads) k_dc(JpegWave w) {
    __shared__ DcSmem sh;
    const uint32_t img = w.spec_list[blockIdx.x / cooperative_groups::this_cluster().num_blocks()];
    const JpegDesc& d = w.descs[img];
    const uint32_t nblocks = d.nblocks;
    const uint32_t* diff = w.diff + d.block_off;
    uint32_t* info = w.info + d.block_off;
    const uint32_t bpm = d.bpm;
    wait_for_previous();
    const auto blocks = [&] { return min(w.cells[d.cell_off].y, nblocks); };
    switch (bpm) {
        case 1: dc_image<1>(diff, info, nblocks, blocks, sh); break;
        case 3: dc_image<3>(diff, info, nblocks, blocks, sh); break;
        case 4: dc_image<4>(diff, info, nblocks, blocks, sh); break;
        default: dc_image<6>(diff, info, nblocks, blocks, sh); break;
    }
}

// Stage-by-stage parity tests look at whole coefficient blocks: fills in the rows the class left out and the DC term.
__global__ void __launch_bounds__(256) k_whole_blocks(JpegWave w, uint32_t nblocks) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x, blk = i >> 3, row = i & 7u;
    wait_for_previous();
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
template <int CELL>
void allow_cells(size_t most) {
    allow_smem(k_huff_guess<CELL, false>, most - 4096);  // (it has static arrays as well)
    allow_smem(k_huff_guess<CELL, true>, most - 4096);
    allow_smem(k_huff_chain<256, CELL, false>, most);
    allow_smem(k_huff_chain<1024, CELL, false>, most);
    allow_smem(k_huff_chain<1024, CELL, true>, most);
    allow_smem(k_huff_write<kDecodeThreads, CELL>, most);
    allow_smem(k_huff_write<kDecodeThreadsMany, CELL>, most);
}

// Dynamic shared memory beyond the default limit has to be allowed once per device and kernel.
void configure_once() {
    static std::once_flag done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    std::call_once(done[dev], [] {
        const size_t most = 227 * 1024 - 1024;
        allow_cells<kCellBits>(most);
        allow_cells<kShortCellBits>(most);
        allow_smem(k_huff_restart<kDecodeThreads>, most);
        allow_smem(k_huff_restart<kDecodeThreadsMany>, most);
    });
}

template <int CELL>
void launch_guess(const JpegWave& w, cudaStream_t s) {
    // the cell before the first, the cells, and what a block may run over
    const size_t rows = 1 + (size_t)guess_spans(1, w.guess_span) * w.guess_span + Staged<CELL>::kRowsBehind;
    const size_t smem = rows * Staged<CELL>::kPitch + w.max_pairs * 2 * sizeof(SyncTab);
    if (w.mixed) launch_after(k_huff_guess<CELL, true>, w.guess_ctas.total, kGuessThreads, smem, s, w);
    else launch_after(k_huff_guess<CELL, false>, w.guess_ctas.total, kGuessThreads, smem, s, w);
}

template <int CELL>
void launch_chain(const JpegWave& w, cudaStream_t s) {
    const size_t tables = w.max_pairs * 2 * sizeof(SyncTab);
    if (w.chain_threads == 256) launch_after(k_huff_chain<256, CELL, false>, w.n_spec, 256, sizeof(ChainMisc<256>) + tables, s, w);
    else if (w.mixed) launch_after(k_huff_chain<1024, CELL, true>, w.n_spec, 1024, sizeof(ChainMisc<1024>) + tables, s, w);
    else launch_after(k_huff_chain<1024, CELL, false>, w.n_spec, 1024, sizeof(ChainMisc<1024>) + tables, s, w);
}

template <int T, int CELL>
void launch_write(const JpegWave& w, cudaStream_t s) {
    const size_t smem = sizeof(ValueMisc<T>) + (size_t)(T + Staged<CELL>::kRowsBehind) * Staged<CELL>::kPitch + w.max_pairs * 2 * sizeof(ValueTab);
    launch_after(k_huff_write<T, CELL>, w.write_ctas.total, T, smem, s, w);
}
template <int CELL>
void launch_write(const JpegWave& w, cudaStream_t s) {
    if (w.write_cells == kDecodeThreads) launch_write<kDecodeThreads, CELL>(w, s);
    else launch_write<kDecodeThreadsMany, CELL>(w, s);
}

template <int T>
void launch_restart(const JpegWave& w, cudaStream_t s) {
    launch_after(k_huff_restart<T>, w.restart_ctas.total, T, sizeof(ValueMisc<T>) + kRestartStage<T> + w.max_pairs * 2 * sizeof(ValueTab), s, w);
}

// CTAs per image: eight while they all run at once; with many images that only adds CTAs (1024 files: passes of 3 200 us with two to
// four, 3 189 with one).
void launch_dc(const JpegWave& w, cudaStream_t s) {
    const uint32_t size = w.n_spec <= kSms / 4 ? 8 : w.n_spec <= kSms ? 2 : 1;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = size; attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t at{};
    at.gridDim = dim3(w.n_spec * size); at.blockDim = dim3(kDcThreads); at.stream = s;
    at.attrs = attrs; at.numAttrs = 2;
    cudaLaunchKernelEx(&at, k_dc, w);
}

}  // namespace

void launch_huff_guess(const JpegWave& w, cudaStream_t s) {
    if (!w.guess_ctas.total) return;
    configure_once();
    if (w.cell_bits == (uint32_t)kCellBits) launch_guess<kCellBits>(w, s);
    else launch_guess<kShortCellBits>(w, s);
}

void launch_huff_chain(const JpegWave& w, cudaStream_t s) {
    if (!w.n_spec) return;
    configure_once();
    if (w.cell_bits == (uint32_t)kCellBits) launch_chain<kCellBits>(w, s);
    else launch_chain<kShortCellBits>(w, s);
}

void launch_huff_write(const JpegWave& w, cudaStream_t s) {
    if (!w.n_spec) return;
    configure_once();
    if (w.write_ctas.total) {  // (streams may be empty)
        if (w.cell_bits == (uint32_t)kCellBits) launch_write<kCellBits>(w, s);
        else launch_write<kShortCellBits>(w, s);
    }
    launch_dc(w, s);
}

void launch_huff_restart(const JpegWave& w, cudaStream_t s) {
    if (!w.restart_ctas.total) return;
    configure_once();
    if (w.restart_segs == kDecodeThreads) launch_restart<kDecodeThreads>(w, s);
    else launch_restart<kDecodeThreadsMany>(w, s);
}

void launch_whole_blocks(const JpegWave& w, uint32_t nblocks, cudaStream_t s) {
    if (nblocks) launch_after(k_whole_blocks, (nblocks + 31) / 32, 256, 0, s, w, nblocks);
}

}  // namespace dg
