// Lattice decode: the sync and final passes of streams whose merges bound
// them (every uncaptured plain decode with the planner's own plan, and
// batches).
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
// Measured on GB300, whole decodes, regions and walks -> lattice: 4 KB 151 ->
// 90 us, 128 KB at 3.8 bits per symbol 473 -> 168, 16 MB at 6 bits 324 ->
// 190, 128 MB at 1.5 bits and L = 4096 4139 -> 1255, 256 MB at 0.67 bits
// and L = 4096 2294 -> 998.
#pragma once

#include <cstdint>

#include "mans_device.cuh"
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
constexpr uint32_t kLatSlotsMax = 12;
constexpr uint32_t kLatDead = 15;          // node: no slot at the next block
constexpr uint32_t kLatKeyUsed = 0x80000000u;
constexpr uint32_t kLatEntBits = 21;       // entry: bit offset (8), state index (13)
constexpr uint32_t kLatThreads = 128;      // sync pass
constexpr uint32_t kLatScanThreads = 256;
constexpr uint32_t kLatScanPer = 4;        // blocks per thread of the scan
constexpr uint32_t kLatScanTile = kLatScanThreads * kLatScanPer;
constexpr uint32_t kLatFinalThreads = 256;

struct LatParams {
    const uint32_t* units;
    uint8_t* out;
    const uint32_t* table;          // reference-format table (L words)
    uint32_t* tab_cnt;              // [L] counting table (zero-bit runs folded)
    uint32_t* tab_sym;              // [L] symbol table
    uint32_t* key;                  // [nblk * D] entries (0: free slot)
    uint32_t* node;                 // [nblk * D] count | next slot << 28
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
    uint32_t B;                     // units per block: 4, 8 or 16
    uint32_t nb;                    // blocks between starts
    uint32_t D;                     // slots per block: 4, 8 or 12
    uint32_t nblk;
    uint32_t nseed;
    uint32_t stage_cap;             // final-pass staging bytes per warp
    uint32_t flags;
    uint32_t width;                 // lanes of a sync-pass warp that run trajectories
};

// counters: next start, scan tile ticket, tiles done, longest trajectory
// (blocks), blocks decoded by all trajectories, ~ the first block where the
// true path has no slot
enum : uint32_t {
    kLatNext = 0, kLatTicket = 1, kLatDone = 2, kLatMaxLife = 3, kLatVisits = 4, kLatDeadBlock = 5
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
        if (run + 1 <= kIncMax) {
            const uint32_t t = plain[na[j]];
            p.tab_cnt[j] = ((t & 0xffffu) * 4u) << 16 | ((run + 1) << 8) | ((t >> 16) & 31u);
        } else {
            p.tab_cnt[j] = ((e & 0xffffu) * 4u) << 16 | (1u << 8) | k;
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

__device__ __forceinline__ uint32_t lat_mask4(uint32_t e) {
    uint32_t m;   // k ones from bit 2, k = the low five bits of e
    asm("bmsk.wrap.b32 %0, %1, %2;" : "=r"(m) : "r"(2u), "r"(e));
    return m;
}

// Bit cursor over units in a lane's column of a warp-wide shared tile: unit
// slot i of the lane lies at column + 128 i, so the 32 lanes of a warp read
// 32 different banks wherever their cursors stand.  Units are stored
// shifted up by two bits (the two top bits of the unit before below them):
// the extracted window then holds the code's b at bit 2 and the next
// entry's address is the entry's address field plus the masked window, no
// shift between the lookups.  `pos` counts bits with the slot of the next
// unit a refill takes at (pos >> 5): it is 64 bits ahead of the codeword.
struct LatCursor {
    uint32_t a, e;       // shared address of the current state's entry, the entry
    uint32_t w0, w1;     // shifted units under the cursor
    uint32_t pos;

    // One step; `mask` = (slots - 1) * 128.  Returns the entry stepped over.
    __device__ __forceinline__ uint32_t step(uint32_t col, uint32_t mask) {
        const uint32_t u = lds32(col | ((pos << 2) & mask));
        const uint32_t y = e;
        const uint32_t b4 = __funnelshift_r(w0, w1, pos) & lat_mask4(y);
        a = (y >> 16) + b4;
        e = lds32(a);
        const uint32_t np = __dp4a(y, 1u, pos);   // + byte 0
        const bool r = ((np ^ pos) & 32u) != 0;   // k <= 16: at most one unit
        w0 = r ? w1 : w0;
        w1 = r ? u : w1;
        pos = np;
        return y;
    }
};

// Decodes to the first codeword at or after position `be`, adding the
// codewords stepped over to cnt.  Four steps a test, so the fourth may pass
// the boundary: every step keeps its state in registers of its own and the
// first one past the boundary is taken (a tail loop of single steps costs a
// test per step and, lane against lane, a dozen steps a block).
__device__ __forceinline__ void lat_block(LatCursor& c, uint32_t col, uint32_t mask, uint32_t be,
                                          uint32_t& cnt) {
    LatCursor c0, c1, c2;
    uint32_t n0, n1, n2;
    do {
        cnt = __dp4a(c.step(col, mask), 0x100u, cnt);   // + byte 1
        c0 = c;
        n0 = cnt;
        cnt = __dp4a(c.step(col, mask), 0x100u, cnt);
        c1 = c;
        n1 = cnt;
        cnt = __dp4a(c.step(col, mask), 0x100u, cnt);
        c2 = c;
        n2 = cnt;
        cnt = __dp4a(c.step(col, mask), 0x100u, cnt);
    } while ((int32_t) (be - c.pos) > 0);
    if ((int32_t) (be - c2.pos) <= 0) { c = c2; cnt = n2; }
    if ((int32_t) (be - c1.pos) <= 0) { c = c1; cnt = n1; }
    if ((int32_t) (be - c0.pos) <= 0) { c = c0; cnt = n0; }
}

// ---------------------------------------------------------------------------
// sync pass

__device__ __forceinline__ uint32_t lat_cas(uint32_t* a, uint32_t v) {
    uint32_t r;
    asm volatile("atom.relaxed.gpu.global.cas.b32 %0, [%1], %2, %3;"
                 : "=r"(r) : "l"(a), "r"(0u), "r"(v) : "memory");
    return r;
}

// Loads whose latency a block's decode hides: volatile, so that they are
// issued where they stand and not where their result is first used.
__device__ __forceinline__ uint4 lat_ld_slots(const uint32_t* a) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a));
    return v;
}
__device__ __forceinline__ uint4 lat_ld_units(const uint32_t* a) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a));
    return v;
}

// Takes or finds the slot of entry `val` among slots [from, D) of a block:
// the slots as they are now, four at a time, then a compare-and-swap on the
// first free one.  Returns the slot (kLatDead: none free) and whether a
// trajectory with that entry was there first.
__device__ __forceinline__ uint32_t lat_take(uint32_t* __restrict__ key, uint32_t from, uint32_t D,
                                             uint32_t val, bool& found) {
    found = false;
    uint32_t q = from;
    while (q < D) {
        const uint32_t g = q & ~3u;
        const uint4 k = lat_ld_slots(key + g);
        uint32_t at = g + 4;   // first slot that is free or holds val
        if (k.w == 0 || k.w == val) at = g + 3;
        if (g + 2 >= q && (k.z == 0 || k.z == val)) at = g + 2;
        if (g + 1 >= q && (k.y == 0 || k.y == val)) at = g + 1;
        if (g >= q && (k.x == 0 || k.x == val)) at = g;
        if (at < g + 4) {
            const uint32_t r = lat_cas(key + at, val);
            if (r == 0) return at;
            if (r == val) {
                found = true;
                return at;
            }
            ++at;
        }
        q = at;
    }
    return kLatDead;
}

// The units of block b of a lane into `r` (zero past the end).
template <uint32_t kB>
__device__ __forceinline__ void lat_load_units(uint32_t (&r)[kB], const uint32_t* __restrict__ in,
                                               uint32_t n, uint32_t b) {
    const unsigned long long u = (unsigned long long) b * kB;
    if (u + kB <= n) {
#pragma unroll
        for (uint32_t i = 0; i < kB / 4; ++i) {
            const uint4 x = lat_ld_units(in + u + 4 * i);
            r[4 * i] = x.x; r[4 * i + 1] = x.y; r[4 * i + 2] = x.z; r[4 * i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kB; ++i) r[i] = u + i < n ? __ldg(in + u + i) : 0u;
    }
}

// Stores a block's units, shifted, from unit slot `s` of the lane's column;
// `carry` is the unit before the first, the last unit on return.
template <uint32_t kB>
__device__ __forceinline__ void lat_store_units(const uint32_t (&r)[kB], uint32_t col, uint32_t s,
                                                uint32_t& carry) {
    uint32_t c = carry;
#pragma unroll
    for (uint32_t i = 0; i < kB; ++i) {
        sts32(col + (s + i) * 128, __funnelshift_l(c, r[i], 2));
        c = r[i];
    }
    carry = c;
}

// Shared memory of a sync-pass CTA: the table, then per warp a ring of two
// blocks for every lane, aligned to its size (at most 4 KB).
__host__ __device__ constexpr uint32_t lat_ring_bytes(uint32_t B) { return 2 * B * 128; }

// One lane per trajectory, persistent: a lane whose trajectory ended takes
// the next start.  Bound by the longest trajectory's chain of lookups on
// short streams (57 cycles a step with the block's bookkeeping, 47 for the
// loop alone, against 62 to 83 for the 8-byte entries and a test per step)
// and by the shared-memory lookups (4.5 cycles a warp and step) once 16
// warps run on every SM.  The slots of the next block and the units of the
// one after it are loaded, and a slot is claimed, a block's decode before
// they are needed, which hides their round trips (about 1500 cycles a block
// when they were waited for).
template <uint32_t kB>
__device__ __forceinline__ void lat_sync_body(const LatParams& p) {
    extern __shared__ __align__(16) uint32_t lat_sm[];
    const uint32_t st = *(volatile uint32_t*) p.status;
    if (st & (MANS_DEV_BAD_TABLE | MANS_DEV_DEGENERATE)) return;
    const uint32_t tb = smem_addr(lat_sm);
    lat_load_table(tb, p.tab_cnt, p.L);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr uint32_t kRing = lat_ring_bytes(kB);
    constexpr uint32_t kMask = kRing - 128;          // unit slots of the ring
    constexpr uint32_t kBits = kB * 32;
    const uint32_t col = ((tb + p.L * 4 + kRing - 1) & ~(kRing - 1)) + warp * kRing + lane * 4;
    const uint32_t D = p.D;

    bool on = false, exhausted = false;
    LatCursor c{};
    uint32_t b = 0;             // block the trajectory stands in
    uint32_t be = 0;            // c.pos at the block's end
    uint32_t q = 0;             // its slot there (tentative while `cas` is open)
    uint32_t val = 0, cas = 0;  // the entry at block b and what its compare-and-swap saw
    uint32_t prev = 0;          // node of the block before: its index in the arrays fits 32 bits
    uint32_t pcnt = 0;          // symbols from there to block b
    bool has_prev = false, first = false;   // first: the true start's trajectory
    uint32_t carry = 0, life = 0, max_life = 0, visits = 0;
    uint32_t nx[kB];            // units of block b + 2, in flight

    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !on && lane < p.width);
        if (!exhausted && __popc(idle) >= min(p.width, 8u)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(p.ctr + kLatNext, (uint32_t) __popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            exhausted = base + __popc(idle) >= p.nseed;
            const uint32_t k = base + __popc(idle & ((1u << lane) - 1));
            if (!on && lane < p.width && k < p.nseed) {
                on = true;
                b = k * p.nb;
                first = k == 0;
                const uint32_t rel = first ? p.first_pos : 0u;
                val = kLatKeyUsed | rel | (p.first_idx << 8);
                // the start's own node; a trajectory that came by with the
                // same entry carries on instead
                if (first) {
                    q = 0;
                    p.key[0] = val;
                } else {
                    bool found;
                    q = lat_take(p.key + (size_t) b * D, 1, D, val, found);
                    if (found || q == kLatDead) on = false;
                }
                cas = 0;
                has_prev = false;
                life = 0;
                if (on) {
                    carry = 0;
                    uint32_t r0[kB];
                    lat_load_units<kB>(r0, p.units, p.n_units, b);
                    lat_load_units<kB>(nx, p.units, p.n_units, b + 1);
                    const uint32_t s = (b & 1u) * kB;
                    lat_store_units<kB>(r0, col, s, carry);
                    lat_store_units<kB>(nx, col, s ^ kB, carry);
                    lat_load_units<kB>(nx, p.units, p.n_units, b + 2);
                    c.pos = s * 32 + rel + 64;
                    be = s * 32 + kBits + 64;
                    const uint32_t u0 = s + (rel >> 5);
                    c.w0 = lds32(col | ((u0 * 128) & kMask));
                    c.w1 = lds32(col | (((u0 + 1) * 128) & kMask));
                    c.a = tb + 4 * p.first_idx;
                    c.e = lds32(c.a);
                }
            }
        }
        if (!__any_sync(0xffffffffu, on)) {
            if (exhausted) break;
            continue;
        }
        if (!on) continue;
        // the slots of block b + 1 as they are now, in flight under the decode
        uint4 kn = make_uint4(0, 0, 0, 0);
        const bool more = b + 1 < p.nblk;
        uint32_t* const knext = p.key + (size_t) (b + 1) * D;
        if (more) kn = lat_ld_slots(knext);
        uint32_t cnt = 0;
        if ((int32_t) (be - c.pos) > 0) lat_block(c, col, kMask, be, cnt);
        ++life;
        // the compare-and-swap of block b, issued before the decode
        bool found = false;
        if (cas != 0) {
            if (cas == val) found = true;
            else q = lat_take(p.key + (size_t) b * D, q + 1, D, val, found);
        }
        if (has_prev) p.node[prev] = pcnt | (q << 28);
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
        uint32_t hit = kLatDead;
        if (kn.x == val) hit = 0;
        if (kn.y == val) hit = 1;
        if (kn.z == val) hit = 2;
        if (kn.w == val) hit = 3;
        ++b;
        if (hit != kLatDead) {
            p.node[prev] = pcnt | (hit << 28);
            on = false;
            max_life = max(max_life, life);
            visits += life;
            continue;
        }
        // the true start's trajectory has slot 0 of every block to itself
        q = first ? 0u : (kn.y == 0 ? 1u : (kn.z == 0 ? 2u : 3u));
        cas = lat_cas(knext + q, val);
        // block b + 1 (one ahead again) into the half of the ring that is free
        const uint32_t s = (b & 1u) * kB;      // slots of block b
        lat_store_units<kB>(nx, col, s ^ kB, carry);
        lat_load_units<kB>(nx, p.units, p.n_units, b + 2);
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
// scan: the true path's slot at every block, then its output offsets

// A slot map, one byte a slot: byte s = the slot a node in slot s leads to,
// kLatDead (15, a fixed point) when it leads nowhere; slots from 4 * kW on
// are fixed points too.
template <uint32_t kW>
struct LatMap {
    uint32_t w[kW];
};

template <uint32_t kW>
__device__ __forceinline__ LatMap<kW> lat_identity() {
    LatMap<kW> m;
#pragma unroll
    for (uint32_t i = 0; i < kW; ++i) m.w[i] = 0x03020100u + i * 0x04040404u;
    return m;
}

// g after f: byte permutes by f's bytes within the two halves of g's 16
// entries, then the half by bit 3.
template <uint32_t kW>
__device__ __forceinline__ LatMap<kW> lat_compose(const LatMap<kW>& g, const LatMap<kW>& f) {
    const uint32_t g1 = kW > 1 ? g.w[kW > 1 ? 1 : 0] : 0x07060504u;
    const uint32_t g2 = kW > 2 ? g.w[kW > 2 ? 2 : 0] : 0x0b0a0908u;
    LatMap<kW> h;
#pragma unroll
    for (uint32_t i = 0; i < kW; ++i) {
        const uint32_t x = f.w[i], x7 = x & 0x07070707u;
        const uint32_t sel = __byte_perm((x7 | (x7 >> 4)) & 0x00ff00ffu, 0, 0x4420);
        const uint32_t lo = __byte_perm(g.w[0], g1, sel), hi = __byte_perm(g2, 0x0f0e0d0cu, sel);
        const uint32_t up = ((x >> 3) & 0x01010101u) * 0xffu;
        h.w[i] = (lo & ~up) | (hi & up);
    }
    return h;
}

template <uint32_t kW>
__device__ __forceinline__ uint32_t lat_apply(const LatMap<kW>& m, uint32_t s) {
    uint32_t x = s;
#pragma unroll
    for (uint32_t i = 0; i < kW; ++i)
        if ((s >> 2) == i) x = (m.w[i] >> (8 * (s & 3u))) & 15u;
    return x;
}

// look-back words: four bits a slot (12 slots), the state in bits 56..59
// (bits 62..63 of a sum)
constexpr unsigned long long kLatAgg = 1, kLatInc = 2;

__device__ __forceinline__ unsigned long long lat_ld(const unsigned long long* a) {
    return *(volatile const unsigned long long*) a;
}

// A tile of consecutive blocks in the scan: every thread's kLatScanPer
// blocks, their slot maps, and the composition of the earlier threads' of
// its warp; s_map holds each warp's whole map.
template <uint32_t kD>
struct LatTile {
    static constexpr uint32_t kW = kD / 4;
    static constexpr uint32_t kWarps = kLatScanThreads / 32;
    struct Shared {
        LatMap<kW> map[kWarps];
        unsigned long long sum[kWarps];
        unsigned long long base;
        uint32_t slot, dead;
    };
    LatMap<kW> f[kLatScanPer], exc;
    uint32_t b0;
    uint32_t cnt[kLatScanPer], ent[kLatScanPer];
    unsigned long long sum, run;

    __device__ __forceinline__ void maps(const LatParams& p, Shared& sh, uint32_t first) {
        const uint32_t t = threadIdx.x, lane = t & 31;
        b0 = first + t * kLatScanPer;
        LatMap<kW> inc = lat_identity<kW>();
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            const uint32_t b = b0 + i;
            f[i] = lat_identity<kW>();
            if (b + 1 < p.nblk) {
                const uint4* nd = reinterpret_cast<const uint4*>(p.node + (size_t) b * kD);
#pragma unroll
                for (uint32_t s = 0; s < kW; ++s) {
                    const uint4 v = __ldg(nd + s);   // the top nibbles of four nodes
                    f[i].w[s] = (__byte_perm(__byte_perm(v.x, v.y, 0x0073),
                                             __byte_perm(v.z, v.w, 0x7300), 0x7610) >> 4) & 0x0f0f0f0fu;
                }
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) inc = lat_compose(f[i], inc);
        // inclusive composition over the warp, earlier threads first
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            LatMap<kW> g;
#pragma unroll
            for (uint32_t i = 0; i < kW; ++i) g.w[i] = __shfl_up_sync(0xffffffffu, inc.w[i], o);
            if (lane >= o) inc = lat_compose(inc, g);
        }
        if (lane == 31) sh.map[t >> 5] = inc;
        exc = lat_identity<kW>();
#pragma unroll
        for (uint32_t i = 0; i < kW; ++i) {
            const uint32_t g = __shfl_up_sync(0xffffffffu, inc.w[i], 1);
            if (lane > 0) exc.w[i] = g;
        }
    }

    // With the slot at the tile's first block in sh.slot: the true slot,
    // entry and count at every block of the thread, the warps' count sums,
    // and the first block without a slot (sh.dead, ~0 before).
    __device__ __forceinline__ void path(const LatParams& p, Shared& sh) {
        const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        uint32_t s = sh.slot;
        for (uint32_t w = 0; w < warp; ++w) s = lat_apply(sh.map[w], s);
        s = lat_apply(exc, s);
        sum = 0;
        uint32_t dead = ~0u;
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            const uint32_t b = b0 + i;
            cnt[i] = ent[i] = 0;
            if (b < p.nblk) {
                if (s >= kD) dead = min(dead, b);
                const size_t at = (size_t) b * kD + min(s, kD - 1);
                ent[i] = __ldg(p.key + at) & ((1u << kLatEntBits) - 1);
                if (b + 1 < p.nblk && s < kD) cnt[i] = __ldg(p.node + at) & 0x0fffffffu;
                s = lat_apply(f[i], s);
            }
            sum += cnt[i];
        }
        dead = __reduce_min_sync(0xffffffffu, dead);
        if (lane == 0 && dead != ~0u) atomicMin(&sh.dead, dead);
        run = sum;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const unsigned long long g = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += g;
        }
        if (lane == 31) sh.sum[warp] = run;
    }

    // With the offset of the tile's first block in sh.base.
    __device__ __forceinline__ void store(const LatParams& p, const Shared& sh) {
        unsigned long long o = sh.base + run - sum;
        for (uint32_t w = 0; w < threadIdx.x >> 5; ++w) o += sh.sum[w];
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            if (b0 + i < p.nblk) p.start[b0 + i] = ent[i] | (o << kLatEntBits);
            o += cnt[i];
        }
    }
};

// The true path goes through a block all of whose slots were taken (more
// distinct trajectories than slots): from there one thread decodes it block
// by block until it meets a trajectory that has a slot, and the CTA scans on
// from that node, tile by tile.  Sequential work, so bounded: past
// kLatRepairBlocks (any number on a short stream) the decode reports
// MANS_DEV_SYNC_OVERFLOW.  Run by the last tile to finish.
constexpr uint32_t kLatRepairBlocks = 4096;
constexpr uint32_t kLatRepairUnits = 32768;   // short stream

template <uint32_t kD>
__device__ __noinline__ void lat_repair(const LatParams& p, typename LatTile<kD>::Shared& sh,
                                        uint32_t dead) {
    const unsigned long long bbits = (unsigned long long) p.B * 32;
    uint32_t budget = p.n_units <= kLatRepairUnits ? ~0u : kLatRepairBlocks;
    __shared__ uint32_t s_b;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t b = dead - 1;   // its entry and offset are known
            const volatile unsigned long long* st = p.start;
            unsigned long long v = st[b];
            uint32_t idx = (uint32_t) (v >> 8) & (kMaxStates - 1);
            unsigned long long pos = b * bbits + (v & 255u), off = v >> kLatEntBits;
            uint32_t slot = kLatDead;
            while (slot == kLatDead && budget) {
                while (pos < (b + 1) * bbits) {
                    const uint32_t e = __ldg(p.tab_cnt + idx);
                    const unsigned long long u = pos >> 5;
                    const uint32_t w0 = u < p.n_units ? __ldg(p.units + u) : 0u;
                    const uint32_t w1 = u + 1 < p.n_units ? __ldg(p.units + u + 1) : 0u;
                    const uint32_t bits = __funnelshift_r(w0, w1, (uint32_t) pos & 31u);
                    idx = min((e >> 18) + (bits & ((1u << (e & 31u)) - 1u)), p.L - 1);
                    pos += e & 31u;
                    off += (e >> 8) & 255u;
                }
                ++b;
                --budget;
                if (b >= p.nblk) break;
                const uint32_t ent = (uint32_t) (pos - b * bbits) | (idx << 8);
                p.start[b] = ent | (off << kLatEntBits);
                for (uint32_t q = 0; q < kD; ++q)
                    if (__ldg(p.key + (size_t) b * kD + q) == (ent | kLatKeyUsed)) slot = q;
            }
            s_b = b;
            sh.slot = slot;
            sh.base = off;
            sh.dead = ~0u;
        }
        __syncthreads();
        uint32_t b = s_b;
        if (b >= p.nblk) break;                       // the stream's end
        if (sh.slot == kLatDead) return;              // out of budget
        dead = ~0u;
        for (; b < p.nblk && dead == ~0u; b += kLatScanTile) {
            LatTile<kD> tl;
            tl.maps(p, sh, b);
            __syncthreads();
            tl.path(p, sh);
            __syncthreads();
            tl.store(p, sh);
            dead = sh.dead;
            uint32_t x = sh.slot;
            unsigned long long base = sh.base;
            for (uint32_t w = 0; w < LatTile<kD>::kWarps; ++w) {
                x = lat_apply(sh.map[w], x);
                base += sh.sum[w];
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                sh.slot = x;
                sh.base = base;
            }
            __syncthreads();
        }
        if (dead == ~0u) break;
    }
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAnd(p.status, ~MANS_DEV_SYNC_OVERFLOW);
    }
}

template <uint32_t kD>
__device__ __forceinline__ void lat_scan_body(const LatParams& p, uint32_t tile) {
    using Tile = LatTile<kD>;
    constexpr uint32_t kWarps = Tile::kWarps;
    __shared__ typename Tile::Shared sh;
    const uint32_t st = *(volatile uint32_t*) p.status;
    if (st & (MANS_DEV_BAD_TABLE | MANS_DEV_DEGENERATE)) return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) sh.dead = ~0u;
    Tile tl;
    tl.maps(p, sh, tile * kLatScanTile);
    __syncthreads();
    // the tile's map (lane s follows slot s), then the slot at its first block
    if (warp == 0) {
        uint32_t x = lane & 15u;
        for (uint32_t w = 0; w < kWarps; ++w) x = lat_apply(sh.map[w], x);
        uint32_t slot = 0;   // slot at the tile's first block
        if (tile != 0) {
            const unsigned long long own = lane < kD ? (unsigned long long) x << (4 * lane) : 0ull;
            const unsigned long long agg =
                (unsigned long long) __reduce_or_sync(0xffffffffu, (uint32_t) own) |
                (unsigned long long) __reduce_or_sync(0xffffffffu, (uint32_t) (own >> 32)) << 32;
            if (lane == 0) atomicExch(p.tile_map + tile, agg | (kLatAgg << 56));
            // back over the predecessors, 32 at a time, to the nearest
            // inclusive slot
            uint32_t near = lane & 15u;   // where slot `lane` leads over the tiles passed so far
            int32_t j = (int32_t) tile - 1;
            uint32_t spins = 0;
            for (;;) {
                const int32_t q = j - (int32_t) lane;
                const unsigned long long v = q >= 0 ? lat_ld(p.tile_map + q) : 0ull;
                const uint32_t fl = (uint32_t) (v >> 56) & 15u;
                const uint32_t incl = __ballot_sync(0xffffffffu, q >= 0 && fl == kLatInc);
                const uint32_t stop = incl ? __ffs(incl) - 1 : 31u;
                if (__ballot_sync(0xffffffffu, q >= 0 && fl == 0 && lane <= stop)) {
                    if (++spins > (1u << 22)) {
                        if (lane == 0) atomicOr(p.status, MANS_DEV_SCAN_TIMEOUT);
                        break;
                    }
                    continue;
                }
                // lane s follows slot s (or all the inclusive slot) from the
                // farthest tile to the nearest
                uint32_t r = incl ? (uint32_t) __shfl_sync(0xffffffffu, v, stop) & 15u : (lane & 15u);
                for (int32_t i = (int32_t) stop - (incl ? 1 : 0); i >= 0; --i) {
                    const unsigned long long m = __shfl_sync(0xffffffffu, v, i);
                    if (r < kD) r = (uint32_t) (m >> (4 * r)) & 15u;
                }
                const uint32_t to = __shfl_sync(0xffffffffu, near, r);
                if (incl) {
                    slot = to;
                    break;
                }
                near = to;
                j -= 32;
            }
        }
        const uint32_t end = __shfl_sync(0xffffffffu, x, slot & 15u);
        if (lane == 0) {
            atomicExch(p.tile_map + tile, (unsigned long long) end | (kLatInc << 56));
            sh.slot = slot;
        }
    }
    __syncthreads();
    tl.path(p, sh);
    __syncthreads();
    if (warp == 0) {
        unsigned long long agg = 0;
        for (uint32_t w = 0; w < kWarps; ++w) agg += sh.sum[w];
        unsigned long long pre = 0;
        if (tile != 0) {
            if (lane == 0) atomicExch(p.tile_sum + tile, agg | (kLatAgg << 62));
            int32_t j = (int32_t) tile - 1;
            uint32_t spins = 0;
            for (;;) {
                const int32_t x = j - (int32_t) lane;
                const unsigned long long v = x >= 0 ? lat_ld(p.tile_sum + x) : 0ull;
                const uint32_t fl = (uint32_t) (v >> 62);
                const uint32_t incl = __ballot_sync(0xffffffffu, x >= 0 && fl == kLatInc);
                const uint32_t stop = incl ? __ffs(incl) - 1 : 31u;
                if (__ballot_sync(0xffffffffu, x >= 0 && fl == 0 && lane <= stop)) {
                    if (++spins > (1u << 22)) {
                        if (lane == 0) atomicOr(p.status, MANS_DEV_SCAN_TIMEOUT);
                        break;
                    }
                    continue;
                }
                unsigned long long w = lane <= stop ? v & ~(3ull << 62) : 0ull;
#pragma unroll
                for (uint32_t o = 16; o; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
                pre += w;
                if (incl) break;
                j -= 32;
            }
        }
        if (lane == 0) {
            atomicExch(p.tile_sum + tile, (pre + agg) | (kLatInc << 62));
            sh.base = pre;
        }
    }
    __syncthreads();
    tl.store(p, sh);
    if (threadIdx.x == 0 && sh.dead != ~0u) {
        atomicOr(p.status, MANS_DEV_SYNC_OVERFLOW);
        atomicMax(p.ctr + kLatDeadBlock, ~sh.dead);
    }
    // the last tile repairs a path that ran out of slots
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();   // the CTA's writes, ordered before by the barrier
        const uint32_t ntiles = (p.nblk + kLatScanTile - 1) / kLatScanTile;
        sh.slot = atomicAdd(p.ctr + kLatDone, 1u) == ntiles - 1;
        __threadfence();
    }
    __syncthreads();
    if (!sh.slot) return;
    const uint32_t now = *(volatile uint32_t*) p.status;
    if ((now & MANS_DEV_SYNC_OVERFLOW) && !(now & MANS_DEV_SCAN_TIMEOUT))
        lat_repair<kD>(p, sh, ~*(volatile uint32_t*) (p.ctr + kLatDeadBlock));
}

// ---------------------------------------------------------------------------
// final pass

// Unit slots of a lane's tile in the final pass: the block and at least
// four units of look-ahead, a power of two (the cursor masks its slot).
__host__ __device__ constexpr uint32_t lat_tile_slots(uint32_t B) { return B == 4 ? 8 : 2 * B; }

__device__ __forceinline__ void lat_sts8(uint32_t a, uint32_t v) {
    asm volatile("st.shared.u8 [%0], %1;" :: "r"(a), "r"(v) : "memory");
}

// Bound by the lookups' shared-memory wavefronts (4-byte entries and
// conflict-free unit columns: 16 MB at 6 bits per symbol 29.6 -> 20.9 us).
// The final pass for the warp of blocks g * 32 .. g * 32 + 31, one lane per
// block: the blocks' symbols form one contiguous output range, staged in
// shared memory with the output's 16-byte phase and written with 16-byte
// stores (a range that does not fit is written byte by byte).
template <bool kRev, uint32_t kB>
__device__ __forceinline__ bool lat_final_warp(const LatParams& p, uint32_t tb, uint32_t tile,
                                               uint32_t stage_addr, uint32_t g) {
    extern __shared__ __align__(16) uint32_t lat_sm[];
    const uint32_t lane = threadIdx.x & 31;
    constexpr uint32_t kMask = (lat_tile_slots(kB) - 1) * 128;
    const uint32_t b0 = g << 5, b = b0 + lane;
    const bool have = b < p.nblk;
    const unsigned long long start = have ? __ldg(p.start + b) : 0ull;
    const uint32_t ent = (uint32_t) start & ((1u << kLatEntBits) - 1);
    const unsigned long long off = start >> kLatEntBits;
    unsigned long long off_nx = max((unsigned long long) p.n_out, off);
    const unsigned long long from_next = __shfl_down_sync(0xffffffffu, off, 1);
    if (b + 1 < p.nblk) off_nx = lane < 31 ? from_next : __ldg(p.start + b + 1) >> kLatEntBits;
    // units: the block's and four more (zero past the end)
    const uint32_t col = tile + lane * 4;
    if (have) {
        uint32_t r[kB + 4];
        const unsigned long long u = (unsigned long long) b * kB;
        if (u + kB + 4 <= p.n_units) {
            const uint4* v = reinterpret_cast<const uint4*>(p.units + u);
#pragma unroll
            for (uint32_t i = 0; i < kB / 4 + 1; ++i) {
                const uint4 x = __ldg(v + i);
                r[4 * i] = x.x; r[4 * i + 1] = x.y; r[4 * i + 2] = x.z; r[4 * i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < kB + 4; ++i) r[i] = u + i < p.n_units ? __ldg(p.units + u + i) : 0u;
        }
        uint32_t carry = 0;
        lat_store_units<kB + 4>(r, col, 0, carry);
    }
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
    if (__any_sync(0xffffffffu, !lane_ok)) {
        if (lane == 0) atomicOr(p.status, MANS_DEV_COUNT_MISMATCH);
        return false;
    }
    const unsigned long long end = min(max(off_nx, off), p.n_out);
    // a valid block holds at most B * 32 + 17 bit positions, each with fewer
    // than L codewords
    const unsigned long long cap_sym = (unsigned long long) (kB * 32 + 17) * p.L;
    const uint32_t cnt = have && off < end ? (uint32_t) min(end - off, cap_sym) : 0u;
    if (have) {
        LatCursor c;
        const uint32_t rel = ent & 0xffu;
        c.a = tb + 4 * min(ent >> 8, p.L - 1);
        c.e = lds32(c.a);
        c.pos = rel + 64;
        c.w0 = lds32(col + (rel >> 5) * 128);
        c.w1 = lds32(col + ((rel >> 5) + 1) * 128);
        const uint32_t pos_cap = kB * 32 + kMaxBits + 1 + 64;
        const uint32_t full = off_nx >= off ? (uint32_t) min(off_nx - off, 0xffffffffull) : 0u;
        uint32_t i = 0;
        if (staged && !kRev) {
            uint32_t q = stage_addr + sb + (uint32_t) (off - wlo);
            for (; i < cnt && (q & 3u) && c.pos < pos_cap; ++i, ++q)
                lat_sts8(q, c.step(col, kMask) >> 8);
            for (; i + 4 <= cnt && c.pos < pos_cap; i += 4, q += 4) {
                const uint32_t y0 = c.step(col, kMask), y1 = c.step(col, kMask);
                const uint32_t y2 = c.step(col, kMask), y3 = c.step(col, kMask);
                sts32(q, __byte_perm(__byte_perm(y0, y1, 0x0051), __byte_perm(y2, y3, 0x5100), 0x7610));
            }
            for (; i < cnt && c.pos < pos_cap; ++i, ++q) lat_sts8(q, c.step(col, kMask) >> 8);
        } else if (staged) {
            // decode index i goes to output n_out - 1 - i: downwards
            uint32_t q = stage_addr + sb + (uint32_t) (p.n_out - 1 - off - wlo);
            for (; i < cnt && (q & 3u) != 3u && c.pos < pos_cap; ++i, --q)
                lat_sts8(q, c.step(col, kMask) >> 8);
            for (; i + 4 <= cnt && c.pos < pos_cap; i += 4, q -= 4) {
                const uint32_t y0 = c.step(col, kMask), y1 = c.step(col, kMask);
                const uint32_t y2 = c.step(col, kMask), y3 = c.step(col, kMask);
                sts32(q - 3, __byte_perm(__byte_perm(y3, y2, 0x0051), __byte_perm(y1, y0, 0x5100), 0x7610));
            }
            for (; i < cnt && c.pos < pos_cap; ++i, --q) lat_sts8(q, c.step(col, kMask) >> 8);
        } else if (!kRev) {
            uint8_t* dst = p.out + off;
            for (; i < cnt && c.pos < pos_cap; ++i) dst[i] = (uint8_t) (c.step(col, kMask) >> 8);
        } else {
            uint8_t* dst = p.out + (p.n_out - 1 - off);
            for (; i < cnt && c.pos < pos_cap; ++i) *(dst - i) = (uint8_t) (c.step(col, kMask) >> 8);
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

// Shared memory of a final-pass CTA: table, unit tiles (aligned to their
// size), staging buffers.
__host__ __device__ constexpr uint32_t lat_final_warp_bytes(uint32_t B) {
    return lat_tile_slots(B) * 128;
}

template <bool kRev, uint32_t kB>
__device__ __forceinline__ void lat_final_body(const LatParams& p, uint32_t cta, uint32_t nctas) {
    extern __shared__ __align__(16) uint32_t lat_sm[];
    const uint32_t st = *(volatile uint32_t*) p.status;
    if (st & MANS_DEV_DEGENERATE) {
        // single-symbol table: every state decodes that symbol
        const uint8_t sym = (uint8_t) (__ldg(p.table) >> 16);
        const unsigned long long stride = (unsigned long long) nctas * blockDim.x;
        for (unsigned long long i = (unsigned long long) cta * blockDim.x + threadIdx.x;
             i < p.n_out; i += stride)
            p.out[i] = sym;
        return;
    }
    if (st & (MANS_DEV_BAD_TABLE | MANS_DEV_SYNC_OVERFLOW | MANS_DEV_SCAN_TIMEOUT)) return;
    const uint32_t tb = smem_addr(lat_sm);
    lat_load_table(tb, p.tab_sym, p.L);
    const uint32_t warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    constexpr uint32_t kTile = lat_final_warp_bytes(kB);
    const uint32_t tiles = (tb + p.L * 4 + kTile - 1) & ~(kTile - 1);
    const uint32_t stage = tiles + nwarp * kTile + warp * (p.stage_cap + 16);
    const uint32_t groups = (p.nblk + 31) >> 5;
    for (uint32_t g = cta * nwarp + warp; g < groups; g += nctas * nwarp)
        if (!lat_final_warp<kRev, kB>(p, tb, tiles + warp * kTile, stage, g)) return;
}

}  // namespace mans
