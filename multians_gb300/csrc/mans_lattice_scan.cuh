// The parts of a lattice pass that the decoder (mans_lattice.cuh) and the
// encoder (mans_encode.cu) share: the slots of a block, and the scan that
// finds the true path through them and its offsets.
//
// P, the parameter block of either, has
//   key    [nblk * D]  entries at each block, bit 31 set (0: free slot)
//   node   [nblk * D]  count of the block (27 bits) | next slot << 27
//   start  [nblk]      out: true entry (kLatEntBits) | offset << kLatEntBits
//   tile_map, tile_sum [ntiles]  look-back words, zero before
//   ctr    [8]         counters, zero before
//   status, nblk
// and, for paths that run out of slots and for the end of the path,
//   uint32_t repair_blocks()       sequential blocks a repair may take
//   uint32_t repair_words()        words of the tables a repair reads, and
//   void repair_load(sm)           the CTA: loads them into the kernel's dynamic
//                                  shared memory sm (lat_scan_smem bytes)
//   void advance(sm, b, ent, off)  one thread: block b from its true entry
//   void finish(slot, off)         one thread: the path's slot and offset at
//                                  the last block
//   void finish_seq(sm, ent, off)  the same where the path has no slot there
#pragma once

#include <cstdint>

#include "multians_gb300.h"

namespace mans {

constexpr uint32_t kLatSlotsMax = 32;
constexpr uint32_t kLatNodeShift = 27;
constexpr uint32_t kLatDead = 31;          // node: no slot at the next block
// Slots that are taken: with 16 and 32 the last one is not, it stands for
// "none" in the scan's maps of four and five bits a slot.
__host__ __device__ constexpr uint32_t lat_none(uint32_t D) { return D > 16 ? 31 : 15; }
__host__ __device__ constexpr uint32_t lat_usable(uint32_t D) {
    return D < lat_none(D) ? D : lat_none(D);
}
constexpr uint32_t kLatKeyUsed = 0x80000000u;
constexpr uint32_t kLatEntBits = 21;       // entry: bit offset (8), state index (13)
constexpr uint32_t kLatScanThreads = 256;
constexpr uint32_t kLatScanPer = 4;        // blocks per thread of the scan
constexpr uint32_t kLatScanTile = kLatScanThreads * kLatScanPer;

// Dynamic shared memory of a scan kernel, used by repairs only.
constexpr size_t lat_scan_smem(size_t repair_words) {
    return (repair_words + 1) / 2 * 8 + kLatScanTile * 8;
}

// counters: next start, scan tile ticket, longest trajectory (blocks), blocks
// decoded by all trajectories, blocks decoded again by repairs
enum : uint32_t { kLatNext = 0, kLatTicket = 1, kLatMaxLife = 3, kLatVisits = 4, kLatRepaired = 5 };

// ---------------------------------------------------------------------------
// slots

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

// Takes or finds the slot of entry `val` among slots [from, end) of a block:
// the slots as they are now, four at a time, then a compare-and-swap on the
// first free one.  Returns the slot (kLatDead: none free) and whether a
// trajectory with that entry was there first.
__device__ __forceinline__ uint32_t lat_take(uint32_t* __restrict__ key, uint32_t from, uint32_t end,
                                             uint32_t val, bool& found) {
    found = false;
    uint32_t q = from;
    while (q < end) {
        const uint32_t g = q & ~3u;
        const uint4 k = lat_ld_slots(key + g);
        uint32_t at = g + 4;   // first slot that is free or holds val
        if (k.w == 0 || k.w == val) at = g + 3;
        if (g + 2 >= q && (k.z == 0 || k.z == val)) at = g + 2;
        if (g + 1 >= q && (k.y == 0 || k.y == val)) at = g + 1;
        if (g >= q && (k.x == 0 || k.x == val)) at = g;
        if (at < min(g + 4, end)) {
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

// ---------------------------------------------------------------------------
// scan: the true path's slot at every block, then its output offsets

// A slot map, one byte a slot: byte s = the slot a node in slot s leads to,
// lat_none (15 or 31, a fixed point) when it leads nowhere; slots from 4 * kW
// on are fixed points too.
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

// g after f: byte permutes by f's bytes within each eight of g's entries,
// then the eight by bits 3 and 4.
template <uint32_t kW>
__device__ __forceinline__ LatMap<kW> lat_compose(const LatMap<kW>& g, const LatMap<kW>& f) {
    constexpr uint32_t kAll = kW > 4 ? 8 : 4;
    uint32_t t[kAll];
#pragma unroll
    for (uint32_t i = 0; i < kAll; ++i) t[i] = i < kW ? g.w[i < kW ? i : 0] : 0x03020100u + i * 0x04040404u;
    LatMap<kW> h;
#pragma unroll
    for (uint32_t i = 0; i < kW; ++i) {
        const uint32_t x = f.w[i], x7 = x & 0x07070707u;
        const uint32_t sel = __byte_perm((x7 | (x7 >> 4)) & 0x00ff00ffu, 0, 0x4420);
        const uint32_t up = ((x >> 3) & 0x01010101u) * 0xffu;
        uint32_t v = (__byte_perm(t[0], t[1], sel) & ~up) | (__byte_perm(t[2], t[3], sel) & up);
        if (kW > 4) {
            const uint32_t v2 = (__byte_perm(t[kAll - 4], t[kAll - 3], sel) & ~up) |
                                (__byte_perm(t[kAll - 2], t[kAll - 1], sel) & up);
            const uint32_t far = ((x >> 4) & 0x01010101u) * 0xffu;
            v = (v & ~far) | (v2 & far);
        }
        h.w[i] = v;
    }
    return h;
}

template <uint32_t kW>
__device__ __forceinline__ uint32_t lat_apply(const LatMap<kW>& m, uint32_t s) {
    uint32_t x = s;
#pragma unroll
    for (uint32_t i = 0; i < kW; ++i)
        if ((s >> 2) == i) x = (m.w[i] >> (8 * (s & 3u))) & 31u;
    return x;
}

// look-back words: four bits a slot (15 slots; none with more), the state in
// bits 62..63
constexpr unsigned long long kLatAgg = 1;     // the tile's map or sum
constexpr unsigned long long kLatInc = 2;     // the slot at, or the sum to, its end
constexpr unsigned long long kLatGhost = 3;   // the entry at its end, which has no slot

__device__ __forceinline__ unsigned long long lat_ld(const unsigned long long* a) {
    return *(volatile const unsigned long long*) a;
}

// A tile of consecutive blocks: every thread's kLatScanPer blocks, their slot
// maps, and the composition of the earlier threads' of its warp; sh.map holds
// each warp's whole map.
template <class P, uint32_t kD>
struct LatTile {
    static constexpr uint32_t kW = kD / 4;
    static constexpr uint32_t kNone = lat_none(kD);
    static constexpr uint32_t kWarps = kLatScanThreads / 32;
    struct Shared {
        LatMap<kW> map[kWarps];
        unsigned long long sum[kWarps];
        unsigned long long base;
        uint32_t slot;     // at the tile's first block (kNone: none)
        uint32_t ghost;    // its entry where the path has no slot there (~0: it has)
        uint32_t dead;     // first block without a slot (~0: none)
        uint32_t from;     // the path is followed from this block
        uint32_t end;      // slot after the tile
    };
    LatMap<kW> f[kLatScanPer], exc;
    uint32_t b0, last;   // last: the slot at the stream's last block (kNone: not here)
    uint32_t cnt[kLatScanPer], ent[kLatScanPer];
    unsigned long long sum, run;

    __device__ __forceinline__ void load(const P& p, uint32_t first) {
        b0 = first + threadIdx.x * kLatScanPer;
        last = kNone;
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            const uint32_t b = b0 + i;
            cnt[i] = ent[i] = 0;
            f[i] = lat_identity<kW>();
            if (b + 1 < p.nblk) {
                const uint4* nd = reinterpret_cast<const uint4*>(p.node + (size_t) b * kD);
#pragma unroll
                for (uint32_t s = 0; s < kW; ++s) {
                    const uint4 v = __ldg(nd + s);   // the top five bits of four nodes
                    f[i].w[s] = (__byte_perm(__byte_perm(v.x, v.y, 0x0073),
                                             __byte_perm(v.z, v.w, 0x7300), 0x7610) >> 3) &
                                (kNone * 0x01010101u);
                }
                if (kD > kNone) f[i].w[kW - 1] |= kNone << 24;   // the slot that stands for none
            }
        }
    }

    // Inclusive composition over the warp, earlier threads first.
    __device__ __forceinline__ void scan(Shared& sh) {
        const uint32_t lane = threadIdx.x & 31;
        LatMap<kW> inc = lat_identity<kW>();
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) inc = lat_compose(f[i], inc);
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            LatMap<kW> g;
#pragma unroll
            for (uint32_t i = 0; i < kW; ++i) g.w[i] = __shfl_up_sync(0xffffffffu, inc.w[i], o);
            if (lane >= o) inc = lat_compose(inc, g);
        }
        if (lane == 31) sh.map[threadIdx.x >> 5] = inc;
        exc = lat_identity<kW>();
#pragma unroll
        for (uint32_t i = 0; i < kW; ++i) {
            const uint32_t g = __shfl_up_sync(0xffffffffu, inc.w[i], 1);
            if (lane > 0) exc.w[i] = g;
        }
    }

    // With the slot at the tile's first block in sh.slot: the true slot,
    // entry and count at every block of the thread from sh.from on, and the
    // first block without a slot (sh.dead, ~0 before).
    __device__ __forceinline__ void path(const P& p, Shared& sh) {
        const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        uint32_t s = sh.slot;
        for (uint32_t w = 0; w < warp; ++w) s = lat_apply(sh.map[w], s);
        s = lat_apply(exc, s);
        uint32_t dead = ~0u;
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            const uint32_t b = b0 + i;
            if (b < p.nblk && b >= sh.from) {
                const bool ok = s < lat_usable(kD);
                if (!ok) dead = min(dead, b);
                const size_t at = (size_t) b * kD + min(s, kD - 1);
                ent[i] = __ldg(p.key + at) & ((1u << kLatEntBits) - 1);
                cnt[i] = b + 1 < p.nblk && ok ? __ldg(p.node + at) & ((1u << kLatNodeShift) - 1) : 0u;
                if (b + 1 == p.nblk) last = s;
            }
            s = lat_apply(f[i], s);
        }
        dead = __reduce_min_sync(0xffffffffu, dead);
        if (lane == 0 && dead != ~0u) atomicMin(&sh.dead, dead);
        if (threadIdx.x == kLatScanThreads - 1) sh.end = s;
    }

    // The warps' count sums.
    __device__ __forceinline__ void sums(Shared& sh) {
        const uint32_t lane = threadIdx.x & 31;
        sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) sum += cnt[i];
        run = sum;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const unsigned long long g = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += g;
        }
        if (lane == 31) sh.sum[threadIdx.x >> 5] = run;
    }

    // With the offset of the tile's first block in sh.base.
    __device__ __forceinline__ void store(const P& p, const Shared& sh) {
        unsigned long long o = sh.base + run - sum;
        for (uint32_t w = 0; w < threadIdx.x >> 5; ++w) o += sh.sum[w];
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            if (b0 + i < p.nblk) p.start[b0 + i] = ent[i] | (o << kLatEntBits);
            if (b0 + i + 1 == p.nblk && last < lat_usable(kD)) p.finish(last, o);
            o += cnt[i];
        }
    }
};

// The true path enters the tile without a slot (sh.ghost: its entry there) or
// goes through a block all of whose slots were taken (sh.dead): more distinct
// trajectories than slots.  One thread decodes on from there block by block
// until it meets a trajectory that has a slot, the tile is followed from
// that node, and so on to its end.  Sequential work, so bounded: past
// repair_blocks() over the whole stream the path is given up
// (MANS_DEV_SYNC_OVERFLOW), at once and not at the end of a stretch (16 M of
// two symbols, L = 4096: 1024 blocks in one stretch, 38 ms).  Later tiles wait for this one's end as always.
template <class P, uint32_t kD>
__device__ __noinline__ void lat_repair(const P& p, LatTile<P, kD>& tl,
                                        typename LatTile<P, kD>::Shared& sh, uint32_t first) {
    extern __shared__ __align__(16) uint32_t lat_repair_sm[];
    // entry and count of the blocks decoded here
    uint2* const s_over = reinterpret_cast<uint2*>(lat_repair_sm + ((p.repair_words() + 1) & ~1u));
    __shared__ uint32_t s_at, s_ent;
    constexpr uint32_t kNone = lat_none(kD);
    const uint32_t stop = min(first + kLatScanTile, p.nblk);
    p.repair_load(lat_repair_sm);
    uint32_t b = first;          // the sequential stretch starts here
    uint32_t ent = sh.ghost;     // with this entry
    bool known = ent != ~0u;
    for (;;) {
        if (!known) {
            // from the last block that has a slot
            b = sh.dead - 1;
#pragma unroll
            for (uint32_t i = 0; i < kLatScanPer; ++i)
                if (tl.b0 + i == b) s_ent = tl.ent[i];
            __syncthreads();
            ent = s_ent;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t x = b, e = ent, slot = kNone;
            const uint32_t had = *(volatile uint32_t*) (p.ctr + kLatRepaired);
            const uint32_t left = p.repair_blocks() > had ? p.repair_blocks() - had : 0;
            while (x < stop && x - b <= left) {
                unsigned long long n = 0;
                s_over[x - first].x = e;
                if (x + 1 < p.nblk) p.advance(lat_repair_sm, x, e, n);
                s_over[x - first].y = (uint32_t) n;
                if (++x >= stop) break;
                const uint4* keys = reinterpret_cast<const uint4*>(p.key + (size_t) x * kD);
                const uint32_t want = e | kLatKeyUsed;
#pragma unroll
                for (uint32_t w = 0; w < kD / 4; ++w) {
                    const uint4 k = __ldg(keys + w);
                    if (k.x == want) slot = 4 * w;
                    if (k.y == want) slot = 4 * w + 1;
                    if (k.z == want) slot = 4 * w + 2;
                    if (k.w == want) slot = 4 * w + 3;
                }
                if (slot != kNone) break;
            }
            const uint32_t used = atomicAdd(p.ctr + kLatRepaired, x - b) + (x - b);
            if (used > p.repair_blocks()) {
                atomicOr(p.status, MANS_DEV_SYNC_OVERFLOW);
                slot = kNone;
                e = ~0u;
            }
            s_at = x;
            sh.ghost = slot == kNone ? e : ~0u;   // leaves the tile without a slot
            sh.end = slot;
            sh.dead = ~0u;
            sh.from = x;
            sh.slot = slot;
        }
        __syncthreads();
        const uint32_t at = s_at, slot = sh.slot;
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            const uint32_t x = tl.b0 + i;
            if (x >= b && x < at) {
                tl.ent[i] = s_over[x - first].x;
                tl.cnt[i] = s_over[x - first].y;
                if (x + 1 == p.nblk) tl.last = kLatSlotsMax;   // the end, without a slot
            }
        }
        if (slot == kNone) break;   // at the tile's end, or given up
        // follow the tile from block `at`: the blocks before it lead there
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i)
            if (tl.b0 + i < at)
#pragma unroll
                for (uint32_t w = 0; w < kD / 4; ++w) tl.f[i].w[w] = slot * 0x01010101u;
        tl.scan(sh);
        __syncthreads();
        tl.path(p, sh);
        __syncthreads();
        const bool dead = sh.dead != ~0u, end = sh.end == kNone;
        __syncthreads();
        if (!dead && !end) break;
        // the last block leads to one without a slot: the next tile's
        if (!dead && threadIdx.x == 0) sh.dead = stop;
        known = false;
        __syncthreads();
    }
    __syncthreads();
}

template <class P, uint32_t kD>
__device__ __forceinline__ void lat_scan_body(const P& p, uint32_t tile) {
    using Tile = LatTile<P, kD>;
    constexpr uint32_t kWarps = Tile::kWarps, kNone = Tile::kNone;
    __shared__ typename Tile::Shared sh;
    const uint32_t st = *(volatile uint32_t*) p.status;
    if (st & (MANS_DEV_BAD_TABLE | MANS_DEV_DEGENERATE)) return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = tile * kLatScanTile;
    if (threadIdx.x == 0) {
        sh.dead = ~0u;
        sh.from = first;
    }
    Tile tl;
    tl.load(p, first);
    tl.scan(sh);
    __syncthreads();
    // the tile's map (lane s follows slot s), then the slot at its first block
    if (warp == 0) {
        uint32_t x = lane & kNone;
        for (uint32_t w = 0; w < kWarps; ++w) x = lat_apply(sh.map[w], x);
        uint32_t slot = 0, ghost = ~0u;
        if (tile != 0 && kD > 16) {
            // a map does not fit a look-back word: the tile before's end
            uint32_t spins = 0;
            for (;;) {
                const unsigned long long v = lat_ld(p.tile_map + tile - 1);
                if ((v >> 62) >= kLatInc) {
                    const bool is_ghost = (v >> 62) == kLatGhost;
                    if (is_ghost) ghost = (uint32_t) v & ((1u << kLatEntBits) - 1);
                    slot = is_ghost ? kNone : (uint32_t) v & kNone;
                    break;
                }
                if (++spins > (1u << 24)) {
                    if (lane == 0) atomicOr(p.status, MANS_DEV_SCAN_TIMEOUT);
                    slot = kNone;
                    break;
                }
            }
            slot = __shfl_sync(0xffffffffu, slot, 0);
            ghost = __shfl_sync(0xffffffffu, ghost, 0);
        } else if (tile != 0) {
            const unsigned long long own =
                lane < lat_usable(kD) ? (unsigned long long) x << (4 * lane) : 0ull;
            const unsigned long long agg =
                (unsigned long long) __reduce_or_sync(0xffffffffu, (uint32_t) own) |
                (unsigned long long) __reduce_or_sync(0xffffffffu, (uint32_t) (own >> 32)) << 32;
            if (lane == 0) atomicExch(p.tile_map + tile, agg | (kLatAgg << 62));
            // back over the predecessors, 32 at a time, to the nearest whose
            // end is known
            uint32_t near = lane & 15u;   // where slot `lane` leads over the tiles passed so far
            int32_t j = (int32_t) tile - 1;
            uint32_t spins = 0;
            for (;;) {
                const int32_t q = j - (int32_t) lane;
                const unsigned long long v = q >= 0 ? lat_ld(p.tile_map + q) : 0ull;
                const uint32_t fl = (uint32_t) (v >> 62);
                const uint32_t incl = __ballot_sync(0xffffffffu, q >= 0 && fl >= kLatInc);
                const uint32_t stop = incl ? __ffs(incl) - 1 : 31u;
                bool wait = __any_sync(0xffffffffu, q >= 0 && fl == 0 && lane <= stop);
                if (!wait) {
                    const unsigned long long e = __shfl_sync(0xffffffffu, v, stop);
                    const bool is_ghost = incl && (e >> 62) == kLatGhost;
                    // lane s follows slot s (or all the known one) from the
                    // farthest tile to the nearest
                    uint32_t r = incl ? (uint32_t) e & 15u : (lane & 15u);
                    for (int32_t i = (int32_t) stop - (incl ? 1 : 0); i >= 0; --i) {
                        const unsigned long long m = __shfl_sync(0xffffffffu, v, i);
                        if (r < lat_usable(kD)) r = (uint32_t) (m >> (4 * r)) & 15u;
                    }
                    const uint32_t to = __shfl_sync(0xffffffffu, near, r);
                    if (!incl) {
                        near = to;
                        j -= 32;
                        continue;
                    }
                    const bool direct = j == (int32_t) tile - 1 && stop == 0;
                    if (direct) {   // the tile before: its end, whatever it is
                        if (is_ghost) ghost = (uint32_t) e & ((1u << kLatEntBits) - 1);
                        slot = is_ghost ? kNone : (uint32_t) e & 15u;
                        break;
                    }
                    if (!is_ghost && to != kNone) {
                        slot = to;
                        break;
                    }
                    // a path without a slot on the way here: the tile it is
                    // in has to find it first
                    wait = true;
                    near = lane & 15u;
                    j = (int32_t) tile - 1;
                }
                if (++spins > (1u << 24)) {
                    if (lane == 0) atomicOr(p.status, MANS_DEV_SCAN_TIMEOUT);
                    slot = kNone;
                    break;
                }
            }
        }
        const uint32_t end = __shfl_sync(0xffffffffu, x, slot & kNone);
        if (lane == 0) {
            // a path that keeps a slot to the tile's end needs nothing more
            if (end != kNone || (slot == kNone && ghost == ~0u))
                atomicExch(p.tile_map + tile, (unsigned long long) end | (kLatInc << 62));
            sh.slot = slot;
            sh.ghost = ghost;
            sh.end = end;
        }
    }
    __syncthreads();
    const bool lost = sh.slot == kNone && sh.ghost == ~0u;   // given up before
    const bool broken = !lost && sh.end == kNone && first + kLatScanTile < p.nblk;
    if (!lost && sh.ghost == ~0u) tl.path(p, sh);
    __syncthreads();
    const bool repair = !lost && (sh.ghost != ~0u || sh.dead != ~0u || broken);
    if (repair) {
        if (threadIdx.x == 0 && sh.ghost == ~0u && sh.dead == ~0u)
            sh.dead = first + kLatScanTile;   // its last block leads to one without a slot
        __syncthreads();
        Tile rt = tl;   // a copy: the call takes its address
        lat_repair<P, kD>(p, rt, sh, first);
        tl = rt;
        if (threadIdx.x == 0)
            atomicExch(p.tile_map + tile,
                       sh.ghost != ~0u ? (unsigned long long) sh.ghost | (kLatGhost << 62)
                                       : (unsigned long long) sh.end | (kLatInc << 62));
    }
    tl.sums(sh);
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
                    if (++spins > (1u << 24)) {
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
    if (repair) {   // a path that ends without a slot
        unsigned long long o = sh.base + tl.run - tl.sum;
        for (uint32_t w = 0; w < warp; ++w) o += sh.sum[w];
        extern __shared__ __align__(16) uint32_t lat_repair_sm[];
#pragma unroll
        for (uint32_t i = 0; i < kLatScanPer; ++i) {
            if (tl.b0 + i + 1 == p.nblk && tl.last == kLatSlotsMax)
                p.finish_seq(lat_repair_sm, tl.ent[i], o);
            o += tl.cnt[i];
        }
    }
}

}  // namespace mans
