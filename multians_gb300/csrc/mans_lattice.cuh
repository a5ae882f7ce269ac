// Lattice decode: the sync and final passes of every plain decode with the
// planner's own plan (but for long streams of eight-bit codes, which symbol
// capture keeps) and of the streams of a batch that fix no geometry, capture or
// seeds.
//
// The stream is cut into blocks of B units.  Trajectories start from a
// guess (bit 0, the stream's first state) every nb blocks, the first one
// from the true start.  At every block start a trajectory looks its entry
// (bit offset, state) up among the entries of the trajectories that have
// been there before: two decodes at the same bit in the same state are
// identical from there on, so on a match it ends, else it takes a free slot
// of the block and goes on.  Every (block, slot) node keeps its entry and,
// once its trajectory has reached the next block, the slot it has there and
// the symbols in between.  The true trajectory is the path from slot 0 of
// block 0: a prefix composition of the blocks' slot maps, then a prefix sum
// of the symbol counts along it.  Then every block's entry and output
// offset are known and the final pass decodes it.
//
// Against walks that wait for one given successor (k_gwalk / k_wwalk), a
// trajectory here ends at the first of ALL others it meets.  With starts
// every s units and a mean pairwise meeting distance T about sqrt(2 T / s)
// distinct ones are under way at any place, so it ends that many times
// sooner and no list of open walks is handed over.  CPU simulation of the
// generator's data, longest chain of dependent steps in units: L = 1024,
// 3.8 bits per symbol, 128 KB: 320 (starts every 16 units) against about
// 1000 (region and walk); L = 4096, 1.5 bits, 32 MB: 1424 (every 64 units)
// against 7000.  The price is work: every unit is decoded sqrt(2 T / s)
// times, so starts are spread no closer than the GPU has idle lanes for.
//
// Measured on GB300, whole decodes, regions and walks -> lattice: 4 KB 144 ->
// 72 us, 128 KB at 3.8 bits per symbol 477 -> 113, 16 MB at 6 bits 353 ->
// 171, 128 MB at 1.5 bits and L = 4096 4340 -> 990, 256 MB at 0.67 bits and
// L = 4096 2621 -> 916; against regions with symbol capture, 256 MB at 6 bits
// 690 -> 536, 512 MB at 8.6 bits 1447 -> 1036.
#pragma once

#include <cstdint>

#include "mans_device.cuh"
#include "mans_lattice_scan.cuh"
#include "mans_tma.cuh"
#include "multians_gb300.h"

namespace mans {

// Prepared table word of the lattice passes, one per state index j:
//   bits 31..16  shared address of the entry of state index base (4 bytes
//                per entry, so b follows at + 4 b)
//   bits 15..8   symbol, or codewords this step stands for
//   bits  7..0   code length k
// Half the size of the 8-byte entry: a 4-byte lookup by 32 lanes takes about
// 3 shared wavefronts against 5, and a CTA's table half the room.
constexpr uint32_t kLatThreads = 128;      // sync pass
constexpr uint32_t kLatFinalThreads = 256;

struct LatParams {
    const uint32_t* units;
    uint8_t* out;
    const uint32_t* table;          // reference-format table (L words)
    uint32_t* tab_cnt;              // [L] counting table (zero-bit runs folded)
    uint32_t* tab_sym;              // [L] symbol table
    uint32_t* key;                  // [nblk * D] entries (0: free slot)
    uint32_t* node;                 // [nblk * D] count | next slot << 27
    unsigned long long* start;      // [nblk] true entry (rel | idx << 8) | output offset << 21
    unsigned long long* tile_map;   // [ntiles] look-back words: slot maps
    unsigned long long* tile_sum;   // [ntiles] look-back words: counts
    uint32_t* ctr;                  // [8] counters
    uint32_t* status;
    unsigned long long n_out;
    uint32_t n_units;
    uint32_t L;
    uint32_t first_idx;
    uint32_t first_pos;
    uint32_t B;                     // units per block: 4, 8, 16 or 32
    uint32_t nb;                    // blocks between starts
    uint32_t D;                     // slots per block: 4, 8, 12, 16 or 32
    uint32_t nblk;
    uint32_t nseed;
    uint32_t stage_cap;             // final-pass staging bytes per warp
    uint32_t flags;
    uint32_t width;                 // lanes of a sync-pass warp that run trajectories

    // scan hooks (mans_lattice_scan.cuh): an entry is the bit offset from the
    // block start and the state index << 8, an offset counts symbols
    // 7 us a block at L = 256, 10 at 1024, up to 37 at 4096.  A blocking call then
    // decodes by regions four times the plan's, which on such data also fail at
    // their plain length and take that long to (L = 1024 3 to 6 ms, L = 4096 9
    // to 18): it loses no time to the lattice.  No stream that plain regions
    // decode was seen to need more (2 to 256 symbols of about equal
    // frequency, L = 8 to 8192, up to 64 MB).  With 4096 blocks 16 M of eight such
    // symbols, L = 1024, took 70 ms a call, by regions alone 32, now 30 (L = 4096:
    // 179, 143, 127).  Short streams are repaired to their end: 600,000 of two
    // symbols 10 ms, by regions 32.
    __device__ __forceinline__ uint32_t repair_blocks() const {
        return n_units <= 32768 ? ~0u : L <= 1024 ? max(L / 4, 128u) : max(L / 8, 256u);
    }
    __device__ __forceinline__ void finish(uint32_t, unsigned long long) const {}
    __device__ __forceinline__ void finish_seq(const uint32_t*, uint32_t, unsigned long long) const {}
    __device__ __forceinline__ uint32_t repair_words() const { return L; }
    __device__ __forceinline__ void repair_load(uint32_t* sm) const {
        for (uint32_t j = threadIdx.x; j < L; j += blockDim.x) sm[j] = __ldg(tab_cnt + j);
    }
    __device__ __forceinline__ void advance(const uint32_t* sm, uint32_t b, uint32_t& ent,
                                            unsigned long long& off) const {
        const auto unit = [&](unsigned long long u) { return u < n_units ? __ldg(units + u) : 0u; };
        uint32_t idx = min(ent >> 8, L - 1), pos = ent & 0xffu;
        unsigned long long u = (unsigned long long) b * B + (pos >> 5);
        uint32_t w0 = unit(u), w1 = unit(u + 1), w2 = unit(u + 2), n = 0;
        while (pos < B * 32) {
            const uint32_t e = sm[idx], k = e & 31u;
            idx = min((e >> 18) + (__funnelshift_r(w0, w1, pos) & ((1u << k) - 1u)), L - 1);
            n += (e >> 8) & 255u;
            if (((pos + k) ^ pos) & 32u) {
                ++u;
                w0 = w1;
                w1 = w2;
                w2 = unit(u + 2);
            }
            pos += k;
        }
        off += n;
        ent = (pos - B * 32) | (idx << 8);
    }
};

// ---------------------------------------------------------------------------
// tables

// Checks and converts the reference table (the rules of prep_body in
// mans_decode.cu) into both lattice tables.  One CTA.
__device__ __forceinline__ void lat_tables(const LatParams& p) {
    extern __shared__ uint32_t lat_sm[];
    const uint32_t L = p.L;
    uint32_t* plain = lat_sm;                    // base | k << 16 | sym << 24
    uint16_t* nxt0 = reinterpret_cast<uint16_t*>(lat_sm + L);
    uint16_t* nxt1 = nxt0 + L;
    uint16_t* z0 = nxt1 + L;
    uint16_t* z1 = z0 + L;
    int bad_l = 0, loop_l = 1, zero_l = 0;

    for (uint32_t j = threadIdx.x; j < L; j += blockDim.x) {
        const uint32_t raw = __ldg(p.table + j);
        const uint32_t ns = raw & 0xffffu, sym = (raw >> 16) & 0xffu, k = raw >> 24;
        bool ok = false, sl = false;
        uint32_t base = 0;
        if (k <= kMaxBits) {
            const uint64_t lo = (uint64_t) ns << k, hi = (uint64_t) (ns + 1) << k;
            if (lo >= L && hi <= 2ull * L) {
                base = (uint32_t) (lo - L);
                ok = k > 0 || base < j;
                sl = k == 0 && base == j;
            }
        }
        uint32_t kk = k;
        if (!ok) { base = 0; kk = 1; }
        bad_l |= ok ? 0 : 1;
        loop_l &= sl ? 1 : 0;
        zero_l |= kk == 0 ? 1 : 0;
        plain[j] = base | (kk << 16) | (sym << 24);
        nxt0[j] = (uint16_t) (kk == 0 ? base : j);
        z0[j] = (uint16_t) (kk == 0 ? 1 : 0);
    }
    const int any_bad = __syncthreads_or(bad_l);
    const int all_loop = __syncthreads_and(loop_l);
    const int any_zero = __syncthreads_or(zero_l);
    if (threadIdx.x == 0)
        *p.status = any_bad ? (all_loop ? MANS_DEV_DEGENERATE : MANS_DEV_BAD_TABLE) : 0u;
    // pointer doubling over the zero-bit runs: nxt -> last state, z -> length
    uint16_t *na = nxt0, *nb = nxt1, *za = z0, *zb = z1;
    if (any_zero)
        for (uint32_t span = 1; span < L; span <<= 1) {
            for (uint32_t j = threadIdx.x; j < L; j += blockDim.x) {
                const uint32_t t = na[j];
                nb[j] = na[t];
                const uint32_t zz = (uint32_t) za[j] + za[t];
                zb[j] = (uint16_t) min(zz, 0xffffu);
            }
            uint16_t* tmp = na; na = nb; nb = tmp;
            tmp = za; za = zb; zb = tmp;
            // every run's end reached: a state whose successor is itself a
            // run member still moves
            int moved = 0;
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < L; j += blockDim.x) moved |= na[na[j]] != na[j];
            if (!__syncthreads_or(moved)) break;
        }
    for (uint32_t j = threadIdx.x; j < L; j += blockDim.x) {
        const uint32_t e = plain[j];
        const uint32_t k = (e >> 16) & 31u;
        p.tab_sym[j] = ((e & 0xffffu) * 4u) << 16 | ((e >> 24) << 8) | k;
        const uint32_t run = za[j];
        if (run < kIncMax) {
            const uint32_t t = plain[na[j]];
            p.tab_cnt[j] = ((t & 0xffffu) * 4u) << 16 | ((run + 1) << 8) | ((t >> 16) & 31u);
        } else {
            // as much of the run as a count holds, no bits (single steps up to
            // there: 1.5 MB with one symbol in 3000 different, L = 4096, 913 us)
            uint32_t t = j;
            for (uint32_t i = 0; i < kIncMax; ++i) t = plain[t] & 0xffffu;
            p.tab_cnt[j] = (t * 4u) << 16 | (kIncMax << 8);
        }
    }
}

// Copies a prepared table into shared memory at shared address tb (a
// multiple of 4, tb + 4 L <= 64 KB), rebasing the entry addresses.
__device__ __forceinline__ void lat_load_table(uint32_t tb, const uint32_t* __restrict__ g,
                                               uint32_t L) {
    const uint32_t add = tb << 16;
    if ((L & 3u) == 0) {
        const uint4* g4 = reinterpret_cast<const uint4*>(g);
        for (uint32_t j = threadIdx.x; j < L / 4; j += blockDim.x) {
            uint4 v = __ldg(g4 + j);
            v.x += add; v.y += add; v.z += add; v.w += add;
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                         :: "r"(tb + j * 16), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
        }
    } else {
        for (uint32_t j = threadIdx.x; j < L; j += blockDim.x)
            sts32(tb + j * 4, __ldg(g + j) + add);
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// cursor

// Shared address of the state after entry e: its address field and 4 b, b = the
// low k bits of window w.  One instruction (k is the low five bits of e)
// instead of a mask and an AND: it lies on the chain from lookup to lookup,
// which is what a trajectory's time consists of.
__device__ __forceinline__ uint32_t lat_next(uint32_t e, uint32_t w) {
    uint32_t b;
    asm("szext.wrap.u32 %0, %1, %2;" : "=r"(b) : "r"(w), "r"(e));
    return (e >> 16) + 4 * b;
}

// Bit cursor over units in a lane's column of a warp-wide shared tile: unit
// slot i of the lane lies at column + 128 i, so the 32 lanes of a warp read
// 32 different banks wherever their cursors stand.  `pos` counts bits with the
// slot of the next unit a refill takes at (pos >> 5): it is 64 bits ahead of
// the codeword.
struct LatCursor {
    uint32_t a, e;       // shared address of the current state's entry, the entry
    uint32_t w0, w1;     // units under the cursor
    uint32_t pos;

    // One step; `mask` = (slots - 1) * 32.  Returns the entry stepped over.
    __device__ __forceinline__ uint32_t step(uint32_t col, uint32_t mask) {
        const uint32_t u = lds32(col + ((pos & mask) << 2));
        const uint32_t y = e;
        a = lat_next(y, __funnelshift_r(w0, w1, pos));
        e = lds32(a);
        const uint32_t np = __dp4a(y, 1u, pos);   // + byte 0
        const bool r = ((np ^ pos) & 32u) != 0;   // k <= 16: at most one unit
        w0 = r ? w1 : w0;
        w1 = r ? u : w1;
        pos = np;
        return y;
    }
};

// The state between the two steps of a pair: the window is the one before
// the pair, `u` the unit a refill takes.
struct LatMid {
    uint32_t a, e, pos, w0, w1, u, base;
    __device__ __forceinline__ void resume(LatCursor& c) const {
        const bool r = ((pos ^ base) & 32u) != 0;
        c.a = a;
        c.e = e;
        c.pos = pos;
        c.w0 = r ? w1 : w0;
        c.w1 = r ? u : w1;
    }
};

// Two steps with one unit load and one refill: the second step's window is
// cut from both units (offset < 32 + 16, code <= 16 bits), and two codes pass
// at most one unit.  Against single steps 4.0 cycles a warp and step
// for 4.5 with the shared pipe full, and half a cycle less alone.
__device__ __forceinline__ void lat_pair(LatCursor& c, uint32_t col, uint32_t mask, uint32_t& y1,
                                         uint32_t& y2, LatMid& m) {
    m.u = lds32(col + ((c.pos & mask) << 2));
    m.w0 = c.w0;
    m.w1 = c.w1;
    m.base = c.pos;
    y1 = c.e;
    m.a = lat_next(y1, __funnelshift_r(c.w0, c.w1, c.pos));
    m.e = lds32(m.a);
    m.pos = __dp4a(y1, 1u, c.pos);
    const uint32_t o = __dp4a(y1, 1u, c.pos & 31u);
    const uint32_t x = (uint32_t) ((((unsigned long long) c.w1 << 32) | c.w0) >> o);
    y2 = m.e;
    c.a = lat_next(y2, x);
    c.e = lds32(c.a);
    c.pos = __dp4a(y2, 1u, m.pos);
    const bool r = ((c.pos ^ m.base) & 32u) != 0;
    c.w0 = r ? m.w1 : m.w0;
    c.w1 = r ? m.u : m.w1;
}

// Decodes to the first codeword at or after position `be`, adding the
// codewords stepped over to cnt.  Two pairs a test, so the last steps may
// pass the boundary: every step keeps its state in registers of its own and
// the first one past the boundary is taken (a tail loop of single steps
// costs a test per step and, lane against lane, a dozen steps a block).
__device__ __forceinline__ void lat_block(LatCursor& c, uint32_t col, uint32_t mask, uint32_t be,
                                          uint32_t& cnt) {
    LatMid m0, m2;
    LatCursor c1;
    uint32_t n0, n1, n2;
    do {
        uint32_t y1, y2;
        lat_pair(c, col, mask, y1, y2, m0);
        n0 = __dp4a(y1, 0x100u, cnt);   // + byte 1
        n1 = __dp4a(y2, 0x100u, n0);
        c1 = c;
        lat_pair(c, col, mask, y1, y2, m2);
        n2 = __dp4a(y1, 0x100u, n1);
        cnt = __dp4a(y2, 0x100u, n2);
    } while ((int32_t) (be - c.pos) > 0);
    if ((int32_t) (be - m2.pos) <= 0) { m2.resume(c); cnt = n2; }
    if ((int32_t) (be - c1.pos) <= 0) { c = c1; cnt = n1; }
    if ((int32_t) (be - m0.pos) <= 0) { m0.resume(c); cnt = n0; }
}

// ---------------------------------------------------------------------------
// sync pass

// Loads of 16 or 32 bytes of units; volatile, so that they are issued where
// they stand, a block ahead.
__device__ __forceinline__ void lat_ld_units(uint32_t* r, const uint32_t* a) {
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(a));
}
__device__ __forceinline__ void lat_ld_units8(uint32_t* r, const uint32_t* a) {
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7]) : "l"(a));
}

// The units of block b of a lane into `r` (zero past the end); wide: the
// stream starts on a 32-byte boundary.  Lanes read apart, so a load costs the
// L1 a pass for every lane whatever its width.
template <uint32_t kB>
__device__ __forceinline__ void lat_load_units(uint32_t (&r)[kB], const uint32_t* __restrict__ in,
                                               uint32_t n, uint32_t b, bool wide) {
    const unsigned long long u = (unsigned long long) b * kB;
    if (u + kB <= n) {
        if (kB >= 8 && wide) {
#pragma unroll
            for (uint32_t i = 0; i < kB / 8; ++i) lat_ld_units8(r + 8 * i, in + u + 8 * i);
        } else {
#pragma unroll
            for (uint32_t i = 0; i < kB / 4; ++i) lat_ld_units(r + 4 * i, in + u + 4 * i);
        }
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kB; ++i) r[i] = u + i < n ? __ldg(in + u + i) : 0u;
    }
}

// Stores units from unit slot `s` of the lane's column.
template <uint32_t kB>
__device__ __forceinline__ void lat_store_units(const uint32_t (&r)[kB], uint32_t col, uint32_t s) {
#pragma unroll
    for (uint32_t i = 0; i < kB; ++i) sts32(col + (s + i) * 128, r[i]);
}

// Shared memory of a sync-pass CTA: the table, then per warp a ring of two
// blocks for every lane.
__host__ __device__ constexpr uint32_t lat_ring_bytes(uint32_t B) { return 2 * B * 128; }

// One lane per trajectory, persistent: a lane whose trajectory ended takes
// the next start, and when there are none left the trajectories of a CTA
// close up into fewer warps (128 MB at 1.5 bits per symbol, L = 4096: sync
// pass 990 -> 893 us; 256 threads a CTA instead of 128: 16 MB 91 -> 106, a
// batch 579 -> 683).  Bound by the longest trajectory's chain of lookups on
// short streams (36 cycles a step, and 1200 to 3000 a block beside its steps;
// 47 a step before the code's bits were cut out by one instruction, 62 to 83
// with 8-byte entries and a test per step)
// and by the L1 data pipe (4.0 passes a warp and step for the lookups, about
// two more for the lanes' own loads of units and slots) once 16 warps run
// on every SM.  The slots of the next block and the units of the
// one after it are loaded, and a slot is claimed, a block's decode before
// they are needed, which hides their round trips (about 1500 cycles a block
// when they were waited for).
// Starts are taken from the counter `next`, up to `limit`.  kNarrow: warps of
// which only p.width lanes run, on inputs with few trajectories; no CTA
// barriers then.  kV: groups of four slots looked at ahead, two in narrow
// warps (a block with more
// than three trajectories costs two exposed round trips otherwise: 146 KB at
// 3.1 bits per symbol, L = 4096, 316 -> 290 us, 128 KB at 3.8 79 -> 67; all
// sixteen looked at: 321 and 73; wide warps: a batch 579 -> 594).
template <uint32_t kB, bool kNarrow, uint32_t kV>
__device__ __forceinline__ void lat_sync_body(const LatParams& p, uint32_t* next, uint32_t limit) {
    extern __shared__ __align__(16) uint32_t lat_sm[];
    __shared__ uint32_t s_live[kLatThreads / 32];
    static_assert(kLatThreads * 28 <= (kLatThreads / 32) * lat_ring_bytes(kB), "states fit the rings");
    const uint32_t st = *(volatile uint32_t*) p.status;
    if (st & (MANS_DEV_BAD_TABLE | MANS_DEV_DEGENERATE)) return;
    const uint32_t tb = smem_addr(lat_sm);
    lat_load_table(tb, p.tab_cnt, p.L);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr uint32_t kRing = lat_ring_bytes(kB);
    constexpr uint32_t kSlots = 2 * kB;              // unit slots of a lane's ring
    constexpr uint32_t kMask = (kSlots - 1) * 32;
    constexpr uint32_t kBits = kB * 32;
    const uint32_t rings = tb + ((p.L * 4 + 15) & ~15u);
    const uint32_t col = rings + warp * kRing + lane * 4;
    const uint32_t D = p.D, end = kV > 2 ? lat_usable(32) : min(D, lat_usable(16));
    const bool wide = ((uintptr_t) p.units & 31) == 0;

    bool on = false, exhausted = false;
    LatCursor c{};
    uint32_t b = 0;             // block the trajectory stands in
    uint32_t be = 0;            // c.pos at the block's end
    uint32_t q = 0;             // its slot there (tentative while `cas` is open)
    uint32_t val = 0, cas = 0;  // the entry at block b and what its compare-and-swap saw
    uint32_t prev = 0;          // node of the block before: its index in the arrays fits 32 bits
    uint32_t pcnt = 0;          // symbols from there to block b
    bool has_prev = false, first = false;   // first: the true start's trajectory
    uint32_t life = 0, max_life = 0, visits = 0;
    uint32_t nx[kB];            // units of block b + 2, in flight
    uint32_t room = blockDim.x; // lanes the CTA's trajectories are spread over

    // the cursor at entry `val` of block b
    const auto begin = [&]() {
        const uint32_t rel = val & 0xffu, s = (b & 1u) * kB;
        if (kB <= 16) {   // both blocks' loads in flight together
            uint32_t r0[kB];
            lat_load_units<kB>(r0, p.units, p.n_units, b, wide);
            lat_load_units<kB>(nx, p.units, p.n_units, b + 1, wide);
            lat_store_units<kB>(r0, col, s);
        } else {
            lat_load_units<kB>(nx, p.units, p.n_units, b, wide);
            lat_store_units<kB>(nx, col, s);
            lat_load_units<kB>(nx, p.units, p.n_units, b + 1, wide);
        }
        lat_store_units<kB>(nx, col, s ^ kB);
        lat_load_units<kB>(nx, p.units, p.n_units, b + 2, wide);
        c.pos = s * 32 + rel + 64;
        be = s * 32 + kBits + 64;
        const uint32_t u0 = s + (rel >> 5);
        c.w0 = lds32(col + (u0 & (kSlots - 1)) * 128);
        c.w1 = lds32(col + ((u0 + 1) & (kSlots - 1)) * 128);
        c.a = tb + 4 * ((val >> 8) & (kMaxStates - 1));
        c.e = lds32(c.a);
    };

    // The CTA's trajectories, false if none is left.
    // No starts left and half the lanes idle: the trajectories move
    // together, into the CTA's first warps (a state is seven words; the
    // units are staged again).  Without it two lanes of three idle.
    const auto close_up = [&]() -> bool {
        const uint32_t n = __syncthreads_count(on);
        if (2 * n <= room && room > 32 && __syncthreads_and(exhausted)) {
            const uint32_t live = __ballot_sync(0xffffffffu, on);
            if (lane == 0) s_live[warp] = __popc(live);
            __syncthreads();
            uint32_t r = __popc(live & ((1u << lane) - 1));
            for (uint32_t w = 0; w < warp; ++w) r += s_live[w];
            if (on) {
                const uint32_t x = rings + r * 28;   // nobody reads the units any more
                sts32(x, b);
                sts32(x + 4, val);
                sts32(x + 8, cas);
                sts32(x + 12, prev);
                sts32(x + 16, pcnt);
                sts32(x + 20, q | (first ? 32u : 0u) | (has_prev ? 64u : 0u));
                sts32(x + 24, life);
            }
            __syncthreads();
            on = threadIdx.x < n;
            if (on) {
                const uint32_t x = rings + threadIdx.x * 28;
                b = lds32(x);
                val = lds32(x + 4);
                cas = lds32(x + 8);
                prev = lds32(x + 12);
                pcnt = lds32(x + 16);
                const uint32_t f = lds32(x + 20);
                q = f & 31u;
                first = (f & 32u) != 0;
                has_prev = (f & 64u) != 0;
                life = lds32(x + 24);
            }
            __syncthreads();
            if (on) begin();
            room = (n + 31) & ~31u;
        }
        return n != 0;
    };

    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !on && lane < p.width);
        if (!exhausted && __popc(idle) >= min(p.width, 8u)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(next, (uint32_t) __popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            exhausted = base + __popc(idle) >= limit;
            const uint32_t k = base + __popc(idle & ((1u << lane) - 1));
            if (!on && lane < p.width && k < limit) {
                on = true;
                b = k * p.nb;
                first = k == 0;
                val = kLatKeyUsed | (first ? p.first_pos : 0u) | (p.first_idx << 8);
                // the start's own node; a trajectory that came by with the
                // same entry carries on instead
                if (first) {
                    q = 0;
                    p.key[0] = val;
                } else {
                    bool found;
                    q = lat_take(p.key + (size_t) b * D, 1, end, val, found);
                    if (found || q == kLatDead) on = false;
                }
                cas = 0;
                has_prev = false;
                life = 0;
                if (on) begin();
            }
        }
        if (kNarrow) {
            if (!__any_sync(0xffffffffu, on)) {
                if (exhausted) break;
                continue;
            }
        } else if (!close_up()) {
            if (__syncthreads_and(exhausted)) break;
            continue;
        }
        if (!on) continue;
        // the slots of block b + 1 as they are now, in flight under the decode
        uint4 kn[kV];
        const bool more = b + 1 < p.nblk;
        uint32_t* const knext = p.key + (size_t) (b + 1) * D;
#pragma unroll
        for (uint32_t g = 0; g < kV; ++g) {
            kn[g] = make_uint4(1, 1, 1, 1);
            if (more && g * 4 < D) kn[g] = lat_ld_slots(knext + g * 4);
        }
        uint32_t cnt = 0;
        if ((int32_t) (be - c.pos) > 0) lat_block(c, col, kMask, be, cnt);
        ++life;
        // the compare-and-swap of block b, issued before the decode
        bool found = false;
        if (cas != 0) {
            if (cas == val) found = true;
            else q = lat_take(p.key + (size_t) b * D, q + 1, end, val, found);
        }
        if (has_prev) p.node[prev] = pcnt | (q << kLatNodeShift);
        if (found || q == kLatDead || !more) {
            on = false;
            max_life = max(max_life, life);
            visits += life;
            continue;
        }
        prev = b * D + q;
        has_prev = true;
        pcnt = cnt;
        // arrive at block b + 1
        val = kLatKeyUsed | (c.pos - be) | (((c.a - tb) << 6));
        uint32_t hit = kLatDead, open = kV == 1 ? 3u : min(kV * 4, D) - 1;
#pragma unroll
        for (uint32_t g = kV; g-- > 0;) {
            if (kn[g].w == val) hit = 4 * g + 3;
            if (kn[g].z == val) hit = 4 * g + 2;
            if (kn[g].y == val) hit = 4 * g + 1;
            if (kn[g].x == val) hit = 4 * g;
            if (kn[g].w == 0) open = 4 * g + 3;
            if (kn[g].z == 0) open = 4 * g + 2;
            if (kn[g].y == 0) open = 4 * g + 1;
            if (kn[g].x == 0 && g > 0) open = 4 * g;
        }
        ++b;
        if (hit != kLatDead) {
            p.node[prev] = pcnt | (hit << kLatNodeShift);
            on = false;
            max_life = max(max_life, life);
            visits += life;
            continue;
        }
        // the true start's trajectory has slot 0 of every block to itself
        q = first ? 0u : open;
        cas = lat_cas(knext + q, val);
        // block b + 1 (one ahead again) into the half of the ring that is free
        const uint32_t s = (b & 1u) * kB;      // slots of block b
        lat_store_units<kB>(nx, col, s ^ kB);
        lat_load_units<kB>(nx, p.units, p.n_units, b + 2, wide);
        if (s == 0) c.pos -= 2 * kBits;
        be = s * 32 + kBits + 64;
    }
    max_life = __reduce_max_sync(0xffffffffu, max_life);
    visits = __reduce_add_sync(0xffffffffu, visits);
    if (lane == 0 && max_life) {
        atomicMax(p.ctr + kLatMaxLife, max_life);
        atomicAdd(p.ctr + kLatVisits, visits);
    }
}

// ---------------------------------------------------------------------------
// final pass

// Units of a warp's 32 blocks in the final pass.  The blocks are one contiguous
// range: it comes in coalesced, as rows of a block each (cp.async of 16 bytes;
// a row loaded by its own lane costs an L1 pass per lane and load: 256 MB at
// 6 bits per symbol 231 -> 217 us, 512 MB at 8.6 500 -> 458), and is then
// turned in place into the cursor's columns (rows read as they are cost
// conflicts as the lanes drift apart: 240 us).  The rows' distance lets lanes
// read 16 bytes of their own row without conflicts; a column holds the block
// and four units of look-ahead.
__host__ __device__ constexpr uint32_t lat_row_words(uint32_t B) { return B == 4 ? 4 : B + 4; }
__host__ __device__ constexpr uint32_t lat_final_warp_bytes(uint32_t B) {
    return 4 * (32 * lat_row_words(B) + 4 > 32 * (B + 4) ? 32 * lat_row_words(B) + 4 : 32 * (B + 4));
}

// Starts the copy of the units of blocks b0 .. b0 + 31 and the four behind
// them into the rows of `tile`, zero past the stream's end.  Streams are
// 16-byte aligned.
template <uint32_t kB>
__device__ __forceinline__ void lat_fill_rows(uint32_t tile, const LatParams& p, uint32_t b0,
                                              uint32_t lane) {
    constexpr uint32_t kPer = kB / 4;   // chunks of four units a row
    const uint64_t u0 = (uint64_t) b0 * kB;
    const auto chunk = [&](uint32_t q) {
        const uint64_t u = u0 + q * 4;
        const uint32_t left = u < p.n_units ? (uint32_t) min((uint64_t) 4, p.n_units - u) : 0u;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     :: "r"(tile + (q / kPer) * (lat_row_words(kB) * 4) + (q % kPer) * 16),
                        "l"(p.units + (left ? u : 0)), "r"(left * 4) : "memory");
    };
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) chunk(i * 32 + lane);
    if (lane == 0) chunk(32 * kPer);
}

// Rows to columns, once the copies have landed.
template <uint32_t kB>
__device__ __forceinline__ void lat_turn_rows(uint32_t tile, uint32_t lane) {
    constexpr uint32_t kRow = lat_row_words(kB) * 4;
    uint32_t r[kB + 4];
    const uint32_t row = tile + lane * kRow;
#pragma unroll
    for (uint32_t i = 0; i < kB + 4; i += 4)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[i]), "=r"(r[i + 1]), "=r"(r[i + 2]), "=r"(r[i + 3])
                     : "r"(i < kB ? row + i * 4 : row + kRow) : "memory");
    __syncwarp();
    lat_store_units<kB + 4>(r, tile + lane * 4, 0);
    __syncwarp();
}

__device__ __forceinline__ void lat_sts8(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u8 [%0], %1;" :: "r"(a), "r"(v) : "memory");
}

// Bound by the lookups' shared-memory wavefronts (4-byte entries and
// conflict-free unit columns: 16 MB at 6 bits per symbol 29.6 -> 20.9 us).
// The final pass for the warp of blocks g * 32 .. g * 32 + 31, one lane per
// block: the blocks' symbols form one contiguous output range, staged in
// shared memory with the output's 16-byte phase and written with 16-byte
// stores.  A range that does not fit (more than 16 KB) is written by its lanes,
// a word at a time (64 served streams, some with blocks of 1500 symbols: 53
// us, by bytes 175).
template <bool kRev, uint32_t kB>
__device__ __forceinline__ bool lat_final_warp(const LatParams& p, uint32_t tb, uint32_t tile,
                                               uint32_t stage_addr, uint32_t g, uint32_t step) {
    extern __shared__ __align__(16) uint32_t lat_sm[];
    const uint32_t lane = threadIdx.x & 31;
    constexpr uint32_t kMask = (2 * kB - 1) * 32;   // no slot wraps
    const uint32_t b0 = g << 5, b = b0 + lane, col = tile + lane * 4;
    const bool have = b < p.nblk;
    lat_fill_rows<kB>(tile, p, b0, lane);
    const unsigned long long start = have ? __ldg(p.start + b) : 0ull;
    const uint32_t ent = (uint32_t) start & ((1u << kLatEntBits) - 1);
    const unsigned long long off = start >> kLatEntBits;
    unsigned long long off_nx = max((unsigned long long) p.n_out, off);
    const unsigned long long from_next = __shfl_down_sync(0xffffffffu, off, 1);
    if (b + 1 < p.nblk) off_nx = lane < 31 ? from_next : __ldg(p.start + b + 1) >> kLatEntBits;
    const unsigned long long off0 = __shfl_sync(0xffffffffu, off, 0);
    const uint32_t last_lane = min(31u, p.nblk - 1 - b0);
    const unsigned long long off_end = __shfl_sync(0xffffffffu, off_nx, last_lane);
    const unsigned long long lo = min(off0, p.n_out);
    const unsigned long long hi = min(max(off_end, off0), p.n_out);
    // the warp writes output indices [wlo, whi) (mirrored in source order)
    const unsigned long long wlo = kRev ? p.n_out - hi : lo;
    const unsigned long long whi = kRev ? p.n_out - lo : hi;
    const uint32_t sb = (uint32_t) (((uintptr_t) p.out + wlo) & 15u);
    const bool staged = whi - wlo + sb <= p.stage_cap;
    const bool lane_ok = !have || (off >= off0 && max(off_nx, off) <= max(off_end, off0));
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (__any_sync(0xffffffffu, !lane_ok)) {
        if (lane == 0) atomicOr(p.status, MANS_DEV_COUNT_MISMATCH);
        return false;
    }
    const unsigned long long end = min(max(off_nx, off), p.n_out);
    // a valid block holds at most B * 32 + 17 bit positions, each with fewer
    // than L codewords
    const unsigned long long cap_sym = (unsigned long long) (kB * 32 + 17) * p.L;
    const uint32_t cnt = have && off < end ? (uint32_t) min(end - off, cap_sym) : 0u;
    __syncwarp();
    lat_turn_rows<kB>(tile, lane);
    // the next group's units and starts on their way into L2 meanwhile
    // (16 warps an SM don't cover the copy's latency: 217 -> 211 us); not those
    // of the last block, which has none where the stream ends with a block (the
    // test written with + 1 on the left: 256 MB at 0.67 bits 270 -> 274 us)
    if ((uint64_t) b + step * 32 < p.nblk - 1) {
        const uint32_t nx = b + step * 32;
        if (kB == 32 || (lane & (32 / kB - 1)) == 0)
            asm volatile("prefetch.global.L2 [%0];" :: "l"(p.units + (uint64_t) nx * kB));
        if ((lane & 15) == 0) asm volatile("prefetch.global.L2 [%0];" :: "l"(p.start + nx));
    }
    if (have) {
        LatCursor c;
        const uint32_t rel = ent & 0xffu;
        c.a = tb + 4 * min(ent >> 8, p.L - 1);
        c.e = lds32(c.a);
        c.pos = rel + 64;
        c.w0 = lds32(col + (rel >> 5) * 128);
        c.w1 = lds32(col + ((rel >> 5) + 1) * 128);
        const uint32_t pos_cap = kB * 32 + kMaxBits + 1 + 64;
        LatMid m;
        const uint32_t full = off_nx >= off ? (uint32_t) min(off_nx - off, 0xffffffffull) : 0u;
        uint32_t i = 0;
        if (staged && !kRev) {
            uint32_t q = stage_addr + sb + (uint32_t) (off - wlo);
            for (; i < cnt && (q & 3u) && c.pos < pos_cap; ++i, ++q)
                lat_sts8(q, c.step(col, kMask) >> 8);
            for (; i + 4 <= cnt && c.pos < pos_cap; i += 4, q += 4) {
                uint32_t y0, y1, y2, y3;
                lat_pair(c, col, kMask, y0, y1, m);
                lat_pair(c, col, kMask, y2, y3, m);
                sts32(q, __byte_perm(__byte_perm(y0, y1, 0x0051), __byte_perm(y2, y3, 0x5100), 0x7610));
            }
            for (; i < cnt && c.pos < pos_cap; ++i, ++q) lat_sts8(q, c.step(col, kMask) >> 8);
        } else if (staged) {
            // decode index i goes to output n_out - 1 - i: downwards
            uint32_t q = stage_addr + sb + (uint32_t) (p.n_out - 1 - off - wlo);
            for (; i < cnt && (q & 3u) != 3u && c.pos < pos_cap; ++i, --q)
                lat_sts8(q, c.step(col, kMask) >> 8);
            for (; i + 4 <= cnt && c.pos < pos_cap; i += 4, q -= 4) {
                uint32_t y0, y1, y2, y3;
                lat_pair(c, col, kMask, y0, y1, m);
                lat_pair(c, col, kMask, y2, y3, m);
                sts32(q - 3, __byte_perm(__byte_perm(y3, y2, 0x0051), __byte_perm(y1, y0, 0x5100), 0x7610));
            }
            for (; i < cnt && c.pos < pos_cap; ++i, --q) lat_sts8(q, c.step(col, kMask) >> 8);
        } else if (!kRev) {
            uint8_t* dst = p.out + off;
            for (; i < cnt && ((uintptr_t) dst & 3u) && c.pos < pos_cap; ++i)
                *dst++ = (uint8_t) (c.step(col, kMask) >> 8);
            for (; i + 4 <= cnt && c.pos < pos_cap; i += 4, dst += 4) {
                uint32_t y0, y1, y2, y3;
                lat_pair(c, col, kMask, y0, y1, m);
                lat_pair(c, col, kMask, y2, y3, m);
                *reinterpret_cast<uint32_t*>(dst) =
                    __byte_perm(__byte_perm(y0, y1, 0x0051), __byte_perm(y2, y3, 0x5100), 0x7610);
            }
            for (; i < cnt && c.pos < pos_cap; ++i) *dst++ = (uint8_t) (c.step(col, kMask) >> 8);
        } else {
            uint8_t* dst = p.out + (p.n_out - 1 - off);
            for (; i < cnt && ((uintptr_t) dst & 3u) != 3u && c.pos < pos_cap; ++i)
                *dst-- = (uint8_t) (c.step(col, kMask) >> 8);
            for (; i + 4 <= cnt && c.pos < pos_cap; i += 4, dst -= 4) {
                uint32_t y0, y1, y2, y3;
                lat_pair(c, col, kMask, y0, y1, m);
                lat_pair(c, col, kMask, y2, y3, m);
                *reinterpret_cast<uint32_t*>(dst - 3) =
                    __byte_perm(__byte_perm(y3, y2, 0x0051), __byte_perm(y1, y0, 0x5100), 0x7610);
            }
            for (; i < cnt && c.pos < pos_cap; ++i) *dst-- = (uint8_t) (c.step(col, kMask) >> 8);
        }
        // a block decoded to its full count ends at the next block start
        if (cnt == full && b + 1 < p.nblk && (c.pos < kB * 32 + 64 || c.pos >= pos_cap))
            atomicOr(p.status, MANS_DEV_COUNT_MISMATCH);
    }
    __syncwarp();
    if (!staged || wlo >= whi) return true;
    // [wlo, whi) from stage[sb + (j - wlo)]; the aligned middle in 16 B words
    const uint8_t* stage = reinterpret_cast<const uint8_t*>(lat_sm) + (stage_addr - tb);
    const uintptr_t base = (uintptr_t) p.out;
    unsigned long long a0 = wlo + ((16 - ((base + wlo) & 15)) & 15);
    unsigned long long a1 = whi - min(whi - wlo, (unsigned long long) ((base + whi) & 15));
    if (a0 > a1) a0 = a1 = whi;
    for (unsigned long long i = wlo + lane; i < a0; i += 32) p.out[i] = stage[sb + (i - wlo)];
    for (unsigned long long i = a1 + lane; i < whi; i += 32) p.out[i] = stage[sb + (i - wlo)];
    const uint4* src = reinterpret_cast<const uint4*>(stage + sb + (a0 - wlo));
    uint4* dst = reinterpret_cast<uint4*>(p.out + a0);
    const uint32_t nvec = (uint32_t) ((a1 - a0) >> 4);
    for (uint32_t v = lane; v < nvec; v += 32) dst[v] = src[v];
    __syncwarp();   // tile and staging are refilled by the next group
    return true;
}

// The CTA's share of an output of one symbol.  Such a stream is one unit long
// and has one CTA, so the stores are as wide as they get (128 MB by bytes 35.5
// ms, so 2.0).  Not inlined: it would cost the batched pass registers (69 -> 80).
__device__ __noinline__ void lat_fill(uint8_t* out, unsigned long long n, uint32_t sym, uint32_t cta,
                                      uint32_t nctas) {
    const uint32_t v = sym * 0x01010101u;
    const unsigned long long stride = (unsigned long long) nctas * blockDim.x;
    const unsigned long long t = (unsigned long long) cta * blockDim.x + threadIdx.x;
    const unsigned long long head = min(n, (unsigned long long) ((16 - ((uintptr_t) out & 15)) & 15));
    const unsigned long long nv = (n - head) >> 4;
    uint4* q = reinterpret_cast<uint4*>(out + head);
    for (unsigned long long i = t; i < nv; i += stride) q[i] = make_uint4(v, v, v, v);
    for (unsigned long long i = t; i < head; i += stride) out[i] = (uint8_t) v;
    for (unsigned long long i = head + 16 * nv + t; i < n; i += stride) out[i] = (uint8_t) v;
}

// Shared memory of a final-pass CTA: table, unit tiles, staging buffers.
template <bool kRev, uint32_t kB>
__device__ __forceinline__ void lat_final_body(const LatParams& p, uint32_t cta, uint32_t nctas) {
    extern __shared__ __align__(16) uint32_t lat_sm[];
    const uint32_t st = *(volatile uint32_t*) p.status;
    if (st & MANS_DEV_DEGENERATE) {
        // single-symbol table: every state decodes that symbol
        lat_fill(p.out, p.n_out, __ldg(p.table) >> 16 & 0xffu, cta, nctas);
        return;
    }
    if (st & (MANS_DEV_BAD_TABLE | MANS_DEV_SYNC_OVERFLOW | MANS_DEV_SCAN_TIMEOUT)) return;
    const uint32_t tb = smem_addr(lat_sm);
    lat_load_table(tb, p.tab_sym, p.L);
    const uint32_t warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    constexpr uint32_t kTile = lat_final_warp_bytes(kB);
    const uint32_t tiles = tb + ((p.L * 4 + 15) & ~15u);
    const uint32_t stage = tiles + nwarp * kTile + warp * (p.stage_cap + 16);
    const uint32_t groups = (p.nblk + 31) >> 5;
    for (uint32_t g = cta * nwarp + warp; g < groups; g += nctas * nwarp)
        if (!lat_final_warp<kRev, kB>(p, tb, tiles + warp * kTile, stage, g, nctas * nwarp)) return;
}

}  // namespace mans
