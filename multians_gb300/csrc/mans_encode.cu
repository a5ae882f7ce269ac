// GPU tANS encoder producing the reference encoder's exact stream
// (src/ans_encoder.cc:13-72: one raw single-state stream, codes packed
// MSB-first into 32-bit units, units then reversed with four zero units of
// padding as CUHDInputBuffer holds them, src/multians_input_buffer.cc:15-30).
//
// Encoding is sequential in the state: x' = next(s, x >> k(s, x)), and the
// code of each byte is the k low bits of x.  But two encodes of the same
// bytes from different states meet after a while and agree from there on,
// so the lattice decode's method carries over (mans_lattice.cuh), with byte
// positions in place of bit positions and the state alone as the entry:
//
//  k_enc_zero  clears the counters, the look-back words and the slots.
//  k_enc_sync  trajectories start from the initial state every S bytes and
//              each ends at the first other one it meets at a block start;
//              every (block, slot) node gets its code bits and the slot it
//              leads to.
//  k_enc_scan  the true path's slot, state and bit offset at every block; at
//              its end the total bit count T, n_units = floor(T / 32) + 1 and
//              first_bit = T mod 32.
//  k_enc_final one lane per block encodes it from its true state and writes
//              the codes at its bit offset, 32 blocks staged in shared memory
//              and copied out in reversed unit order; the last lane adds the
//              bits the reference's flush leaves below the last unit's valid
//              bits (the last byte's code again when it fitted its unit, else
//              the code of byte value 0 past the end).
//
// Tables: the compact encoder table built on the host from the byte
// histogram (mans_host_encode_tables), loaded into shared memory per CTA.
// L is a power of two <= 8192.
//
// Measured on GB300, 64 MB at 3.8 bits per symbol and L = 4096: 359 us sync,
// 31 scan, 109 final; chunks with merge walks took 195 + 1374 us, found their
// slots too few, and again 744 + 1327 + 305 us with longer chunks.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "mans_device.cuh"
#include "mans_lattice_scan.cuh"
#include "mans_tma.cuh"
#include "multians_gb300.h"

namespace mans {
namespace {

constexpr uint32_t kEncThreads = 128;        // sync pass
constexpr uint32_t kEncCtas = 3;             // per SM, of the persistent sync pass
constexpr uint32_t kEncFinalThreads = 256;
constexpr uint32_t kEncSlots = 16;           // a block
constexpr uint32_t kEncSmallBytes = 1u << 20;

struct EncResult {
    unsigned long long total_bits;
    unsigned long long n_units;
    uint32_t first_bit, first_state;
    uint32_t last_code, last_len;          // the last byte's code
};

struct EncEnd {                            // a trajectory's end at the last block
    uint32_t state, bits, code, len;
};

struct EncParams {
    const uint8_t* sym;
    unsigned long long n;
    const uint32_t* blob;                  // global compact table
    uint32_t L, Bs, nb, D, nblk, nseed, width;
    uint32_t* key;
    uint32_t* node;
    unsigned long long* start;
    unsigned long long* tile_map;
    unsigned long long* tile_sum;
    uint32_t* ctr;
    uint32_t* status;
    EncResult* result;
    EncEnd* end;                           // [D] by slot at the last block
    uint32_t* units;
    unsigned long long cap;                // units capacity (words)

    // scan hooks (mans_lattice_scan.cuh): an entry is the state - L, an
    // offset counts bits
    __device__ __forceinline__ uint32_t repair_blocks() const { return n <= 16384 ? ~0u : 64u; }
    __device__ __forceinline__ void set_result(const EncEnd& e, unsigned long long off) const {
        const unsigned long long T = off + e.bits;
        result->total_bits = T;
        result->n_units = T / 32 + 1;
        result->first_bit = (uint32_t) (T & 31);
        result->first_state = e.state;
        result->last_code = e.code;
        result->last_len = e.len;
        if (T / 32 + 1 + 4 > cap) atomicOr(status, MANS_DEV_COUNT_MISMATCH);
    }
    __device__ __forceinline__ void finish(uint32_t slot, unsigned long long off) const {
        set_result(end[slot], off);
    }
    __device__ __forceinline__ uint32_t repair_words() const { return 512 + (L + 1) / 2; }
    __device__ __forceinline__ void repair_load(uint32_t* sm) const {
        for (uint32_t i = threadIdx.x; i < repair_words(); i += blockDim.x) sm[i] = __ldg(blob + i);
    }
    // one block, by one thread
    __device__ __forceinline__ EncEnd block(const uint32_t* sm, uint32_t b, uint32_t ent) const {
        EncEnd e = {L + min(ent, L - 1), 0, 0, 0};
        const unsigned long long i1 = min((unsigned long long) (b + 1) * Bs, n);
        const uint16_t* nx = reinterpret_cast<const uint16_t*>(sm + 512);
        for (unsigned long long i = (unsigned long long) b * Bs; i < i1; ++i) {
            const uint32_t s = sym[i];
            e.len = min((e.state + sm[2 * s]) >> 16, 31u);
            e.code = e.state & ((1u << e.len) - 1u);
            e.bits += e.len;
            const uint32_t next = nx[min(sm[2 * s + 1] + (e.state >> e.len), L - 1)];
            e.state = min(max(next, L), 2 * L - 1);
        }
        return e;
    }
    __device__ __forceinline__ void advance(const uint32_t* sm, uint32_t b, uint32_t& ent,
                                            unsigned long long& off) const {
        const EncEnd e = block(sm, b, ent);
        ent = e.state - L;
        off += e.bits;
    }
    __device__ __forceinline__ void finish_seq(const uint32_t* sm, uint32_t ent,
                                               unsigned long long off) const {
        set_result(block(sm, nblk - 1, ent), off);
    }
};

// Shared tables: per byte value {delta, shared address of the next state of
// x >> k = 0}, then the L next states as uint16; k = (x + delta) >> 16.
// Entries that do not have the table's form (absent bytes, which the data
// does not hold) lead to the first next state with k = 31, so every address
// stays inside the table.
__device__ __forceinline__ void load_enc_tables(uint32_t tb, const uint32_t* __restrict__ blob,
                                                uint32_t L) {
    const uint32_t nx = tb + 256 * 8;
    const uint32_t lg = 31 - __clz(L);
    for (uint32_t v = threadIdx.x; v < 256; v += blockDim.x) {
        const uint32_t delta = __ldg(blob + 2 * v), base = __ldg(blob + 2 * v + 1);
        const uint32_t m = (delta + 0xffffu) >> 16;
        const uint32_t thr = (m << 16) - delta;
        const uint32_t f = m <= lg + 1 ? thr >> m : 0u;
        const uint32_t first = base + f;
        const bool ok = m >= 1 && f >= 1 && f <= L && thr == f << m &&
                        m == lg + 1 - (f > 1 ? 32 - __clz(f - 1) : 0) && first <= L - f;
        sts32(tb + v * 8, ok ? delta : 31u << 16);
        sts32(tb + v * 8 + 4, ok ? nx + base * 2 : nx);
    }
    const uint32_t* g = blob + 512;
    for (uint32_t i = threadIdx.x; i < (L + 1) / 2; i += blockDim.x) {
        const uint32_t w = __ldg(g + i);
        const uint32_t lo = min(max(w & 0xffffu, L), 2 * L - 1), hi = min(max(w >> 16, L), 2 * L - 1);
        sts32(nx + i * 4, lo | hi << 16);
    }
    __syncthreads();
}

__host__ __device__ constexpr uint32_t enc_table_bytes(uint32_t L) {
    return (256 * 8 + ((L + 1) / 2) * 4 + 15) & ~15u;
}

// Table loads: not volatile, so that the byte values' entries, which do not
// depend on the state, are loaded ahead of the chain that does.
__device__ __forceinline__ uint32_t lds_next(uint32_t a) {
    uint32_t v;
    asm("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds_entry(uint32_t a) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// 16 bytes global -> shared, zero-filled past `bytes`.
__device__ __forceinline__ void cp16(uint32_t dst, const uint8_t* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" :: "n"(kLeft) : "memory");
}

// One encode step of byte value s from state x: returns k; x becomes the
// next state.  A chain of add, shift, shift, address and table load: 50
// cycles a byte (the same with the code length chosen by a threshold test on
// x, 60 with both of its shifts started from x at once), 5.8 a warp and byte
// with 16 warps.
__device__ __forceinline__ uint32_t enc_step(uint32_t& x, uint32_t s, uint32_t tb) {
    const uint2 q = lds_entry(tb + s * 8);
    const uint32_t k = (x + q.x) >> 16;
    x = lds_next(q.y + 2 * (x >> k));
    return k;
}

// Copies block b of the source into a lane's row (bytes past the end zero).
template <uint32_t kBs>
__device__ __forceinline__ void enc_fetch(uint32_t row, const EncParams& p, uint32_t b) {
    const unsigned long long i0 = (unsigned long long) b * kBs;
#pragma unroll
    for (uint32_t i = 0; i < kBs / 16; ++i) {
        const unsigned long long at = i0 + 16 * i;
        const uint32_t have = at < p.n ? (uint32_t) min(p.n - at, 16ull) : 0u;
        cp16(row + 16 * i, p.sym + (have ? at : 0), have);
    }
    cp_commit();
}

// Rows padded by 16 bytes, so that the lanes' 16-byte reads spread over all
// banks: two blocks of a lane in the sync pass, one in the final pass.
__host__ __device__ constexpr uint32_t enc_pair_bytes(uint32_t Bs) { return 2 * Bs + 16; }
__host__ __device__ constexpr uint32_t enc_row_bytes(uint32_t Bs) { return Bs + 16; }

// Sync pass: one lane per trajectory, persistent (the flow of
// lat_sync_body in mans_lattice.cuh).  Bound by the longest trajectory's
// chain on small inputs and by shared-memory lookups on large ones.
template <uint32_t kBs>
__global__ void __launch_bounds__(kEncThreads) k_enc_sync(EncParams p) {
    extern __shared__ __align__(16) uint32_t enc_sm[];
    follow_previous();
    const uint32_t tb = smem_addr(enc_sm);
    load_enc_tables(tb, p.blob, p.L);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t row = tb + enc_table_bytes(p.L) + threadIdx.x * enc_pair_bytes(kBs);
    const uint32_t D = p.D, L = p.L;

    bool on = false, exhausted = false;
    uint32_t b = 0, x = 0, q = 0, val = 0, cas = 0, pbits = 0, life = 0, max_life = 0;
    uint32_t* prev = nullptr;   // node of the block before (its index may need more than 32 bits)
    bool has_prev = false, first = false;
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
                x = L;
                val = kLatKeyUsed;
                if (first) {
                    q = 0;
                    p.key[0] = val;
                } else {
                    bool found;
                    q = lat_take(p.key + (size_t) b * D, 1, lat_usable(kEncSlots), val, found);
                    if (found || q == kLatDead) on = false;
                }
                cas = 0;
                has_prev = false;
                life = 0;
                if (on) {
                    cp_wait<0>();
                    enc_fetch<kBs>(row + (b & 1u) * kBs, p, b);
                }
            }
        }
        if (!__any_sync(0xffffffffu, on)) {
            if (exhausted) break;
            continue;
        }
        if (!on) continue;
        uint4 kn = make_uint4(0, 0, 0, 0);
        const bool more = b + 1 < p.nblk;
        uint32_t* const knext = p.key + (size_t) (b + 1) * D;
        if (more) kn = lat_ld_slots(knext);
        // the block after this one on its way while this one is encoded
        enc_fetch<kBs>(row + ((b + 1) & 1u) * kBs, p, more ? b + 1 : b);
        cp_wait<1>();
        const uint32_t src = row + (b & 1u) * kBs;
        uint32_t bits = 0, x_in = x, len = 0;
        if (more) {
            uint4 v = lds128(src);
#pragma unroll 1
            for (uint32_t i = 16; i <= kBs; i += 16) {
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                if (i < kBs) v = lds128(src + i);
#pragma unroll
                for (uint32_t t = 0; t < 16; ++t)
                    bits += enc_step(x, (w[t >> 2] >> (8 * (t & 3))) & 0xffu, tb);
            }
        } else {
            // the last block: as many bytes as there are
            const uint32_t cnt = (uint32_t) (p.n - (unsigned long long) b * kBs);
            for (uint32_t i = 0; i < cnt; ++i) {
                x_in = x;
                len = enc_step(x, (lds32(src + (i & ~3u)) >> (8 * (i & 3))) & 0xffu, tb);
                bits += len;
            }
        }
        ++life;
        bool found = false;
        if (cas != 0) {
            if (cas == val) found = true;
            else q = lat_take(p.key + (size_t) b * D, q + 1, lat_usable(kEncSlots), val, found);
        }
        if (has_prev) *prev = pbits | (q << kLatNodeShift);
        if (found || q == kLatDead || !more) {
            if (!more && !found && q != kLatDead)
                p.end[q] = {x, bits, x_in & ((1u << len) - 1u), len};
            on = false;
            max_life = max(max_life, life);
            continue;
        }
        prev = p.node + (size_t) b * D + q;
        has_prev = true;
        pbits = bits;
        val = kLatKeyUsed | (x - L);
        uint32_t hit = kLatDead;
        if (kn.x == val) hit = 0;
        if (kn.y == val) hit = 1;
        if (kn.z == val) hit = 2;
        if (kn.w == val) hit = 3;
        ++b;
        if (hit != kLatDead) {
            *prev = pbits | (hit << kLatNodeShift);
            on = false;
            max_life = max(max_life, life);
            continue;
        }
        // the true start's trajectory has slot 0 of every block to itself
        q = first ? 0u : (kn.y == 0 ? 1u : (kn.z == 0 ? 2u : 3u));
        cas = lat_cas(knext + q, val);
    }
    cp_wait<0>();
    max_life = __reduce_max_sync(0xffffffffu, max_life);
    if (lane == 0 && max_life) atomicMax(p.ctr + kLatMaxLife, max_life);
}

template <uint32_t kD>
__global__ void __launch_bounds__(kLatScanThreads) k_enc_scan(EncParams p) {
    __shared__ uint32_t s_tile;
    follow_previous();
    if (threadIdx.x == 0) s_tile = atomicAdd(p.ctr + kLatTicket, 1u);
    __syncthreads();
    lat_scan_body<EncParams, kD>(p, s_tile);
}

__global__ void __launch_bounds__(256) k_enc_zero(uint4* a, size_t na, uint32_t* units, size_t nu) {
    follow_previous();
    const size_t stride = (size_t) gridDim.x * blockDim.x;
    const size_t t = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t i = t; i < na; i += stride) a[i] = make_uint4(0, 0, 0, 0);
    // the units (any word alignment): words to the first 16-byte boundary,
    // vectors, the rest
    const size_t head = min(nu, (size_t) ((16 - ((uintptr_t) units & 15)) & 15) / 4);
    const size_t nv = (nu - head) / 4;
    uint4* v = reinterpret_cast<uint4*>(units + head);
    for (size_t i = t; i < nv; i += stride) v[i] = make_uint4(0, 0, 0, 0);
    for (size_t i = t; i < head; i += stride) units[i] = 0;
    for (size_t i = head + nv * 4 + t; i < nu; i += stride) units[i] = 0;
}

__device__ __forceinline__ void red_or_shared(uint32_t a, uint32_t v) {
    asm volatile("red.shared.or.b32 [%0], %1;" :: "r"(a), "r"(v) : "memory");
}

// Unit words a warp's 32 blocks may span.
__host__ __device__ constexpr uint32_t enc_stage_words(uint32_t Bs, uint32_t lg) {
    return (Bs * lg + 2 + 3) & ~3u;
}

// Final pass: a warp per 32 blocks; bound by instruction issue (about 25 a
// byte).  Their source bytes come in coalesced
// (cp.async into padded rows), every lane packs its block's codes MSB-first
// into the warp's staging words (words it shares with a neighbour by atomic
// OR), and the warp writes the words out in reversed unit order, coalesced;
// only its first and last word may be shared with other warps.
template <uint32_t kBs>
__global__ void __launch_bounds__(kEncFinalThreads) k_enc_final(EncParams p) {
    extern __shared__ __align__(16) uint32_t enc_sm[];
    follow_previous();
    if (*(volatile uint32_t*) p.status & (MANS_DEV_SYNC_OVERFLOW | MANS_DEV_SCAN_TIMEOUT |
                                          MANS_DEV_COUNT_MISMATCH))
        return;
    const uint32_t tb = smem_addr(enc_sm);
    load_enc_tables(tb, p.blob, p.L);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const uint32_t lg = 31 - __clz(p.L);
    constexpr uint32_t kRow = enc_row_bytes(kBs);
    const uint32_t words = enc_stage_words(kBs, lg);
    const uint32_t rows = tb + enc_table_bytes(p.L) + warp * (32 * kRow + words * 4);
    const uint32_t stage = rows + 32 * kRow;
    const EncResult res = *p.result;
    const unsigned long long n_units = res.n_units;
    const uint32_t groups = (p.nblk + 31) >> 5;
    for (uint32_t g = blockIdx.x * nwarp + warp; g < groups; g += gridDim.x * nwarp) {
        const uint32_t b = (g << 5) + lane;
        // 32 blocks of source: 16-byte chunks, consecutive lanes consecutive
        const unsigned long long i0 = (unsigned long long) g * 32 * kBs;
#pragma unroll
        for (uint32_t j = 0; j < kBs / 16; ++j) {
            const uint32_t c = j * 32 + lane;
            const unsigned long long at = i0 + 16ull * c;
            const uint32_t have = at < p.n ? (uint32_t) min(p.n - at, 16ull) : 0u;
            cp16(rows + (c / (kBs / 16)) * kRow + (c % (kBs / 16)) * 16, p.sym + (have ? at : 0), have);
        }
        cp_commit();
        const bool live = b < p.nblk;
        const unsigned long long st = live ? __ldg(p.start + b) : 0ull;
        const unsigned long long o = live ? st >> kLatEntBits : res.total_bits;
        const unsigned long long o0 = __shfl_sync(0xffffffffu, o, 0);
        unsigned long long o1 = res.total_bits;
        if ((g + 1) * 32 < p.nblk) o1 = __ldg(p.start + (g + 1) * 32) >> kLatEntBits;
        const unsigned long long u0 = o0 >> 5;
        const uint32_t span = (uint32_t) min(((o1 + 31) >> 5) - u0, (unsigned long long) words);
        for (uint32_t i = lane; i < span; i += 32) sts32(stage + i * 4, 0);
        cp_wait<0>();
        __syncwarp();
        if (live) {
            uint32_t x = p.L + min((uint32_t) st & ((1u << kLatEntBits) - 1), p.L - 1);
            const unsigned long long left = p.n - (unsigned long long) b * kBs;
            const uint32_t cnt = (uint32_t) min(left, (unsigned long long) kBs);
            uint32_t nbits = (uint32_t) o & 31u;
            uint32_t at = stage + (uint32_t) min((o >> 5) - u0, (unsigned long long) words - 1) * 4;
            const uint32_t at_max = stage + (words - 1) * 4;
            bool shared_word = true;   // the first word: other lanes' bits may be in it
            uint32_t hi = 0, lo = 0;   // pending bits, newest at the bottom of lo
            const auto put = [&](uint32_t code, uint32_t len) {
                hi = __funnelshift_lc(lo, hi, len);
                lo = (lo << len) | code;
                nbits += len;
                if (nbits >= 32) {
                    nbits -= 32;
                    const uint32_t w = __funnelshift_rc(lo, hi, nbits);
                    if (shared_word) red_or_shared(at, w);
                    else sts32(at, w);
                    shared_word = false;
                    at = min(at + 4, at_max);
                }
            };
            const uint32_t src = rows + lane * kRow;
            if (cnt == kBs) {
#pragma unroll 1
                for (uint32_t i = 0; i < kBs; i += 16) {
                    const uint4 v = lds128(src + i);
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (uint32_t t = 0; t < 16; ++t) {
                        const uint32_t x0 = x;
                        const uint32_t len = enc_step(x, (w[t >> 2] >> (8 * (t & 3))) & 0xffu, tb);
                        put(x0 & ((1u << len) - 1u), len);
                    }
                }
            } else {
                for (uint32_t i = 0; i < cnt; ++i) {
                    const uint32_t x0 = x;
                    const uint32_t len = enc_step(x, (lds32(src + (i & ~3u)) >> (8 * (i & 3))) & 0xffu, tb);
                    put(x0 & ((1u << len) - 1u), len);
                }
            }
            if (nbits > 0) red_or_shared(at, lo << (32 - nbits));
        }
        __syncwarp();
        // unit u of the forward stream lives at units[n_units - 1 - u]
        for (uint32_t i = lane; i < span; i += 32) {
            const unsigned long long u = u0 + i;
            if (u < n_units) {
                const uint32_t w = lds32(stage + i * 4);
                uint32_t* a = p.units + (n_units - 1 - u);
                if (i == 0 || i + 1 == span) atomicOr(a, w);
                else *a = w;
            }
        }
        __syncwarp();
    }
    // The flush of the reference encoder (src/ans_encoder.cc:40-66): below
    // the last unit's at = T mod 32 valid bits it adds the high bits of one
    // more code when that code reaches 32 - at bits: the last byte's code
    // again when it fitted its unit (at the unit loop's exit it is still the
    // current entry), else the code of byte value 0 (the byte past the end)
    // from the final state.
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t at = (uint32_t) (res.total_bits & 31);
        const unsigned long long P = res.total_bits - res.last_len;   // start of the last code
        uint32_t code = res.last_code, len = res.last_len;
        if ((uint32_t) (P & 31) + len >= 32) {
            const uint32_t dq = __ldg(p.blob);
            if (dq == 0) return;                                // byte 0 absent: zero entry
            len = (res.first_state + dq) >> 16;
            code = res.first_state & ((1u << len) - 1u);
        }
        if (at + len >= 32) atomicOr(p.units, code >> (at + len - 32));   // unit n_units - 1
    }
}

// Bytes of a histogram CTA at least (256 KB: one CTA for 100 KB, 10.8 us, and
// half a wave for 64 MB, 25 us).
constexpr size_t kHistBytes = 16 * 1024;

// Byte histogram: per-CTA counts in shared memory (one copy per warp, so
// lanes of different warps do not contend), merged into 64-bit totals.
__global__ void __launch_bounds__(256) k_hist(const uint8_t* __restrict__ sym,
                                             unsigned long long n,
                                             unsigned long long* __restrict__ hist) {
    __shared__ uint32_t h[8][256];
    for (uint32_t i = threadIdx.x; i < 8 * 256; i += blockDim.x) (&h[0][0])[i] = 0;
    __syncthreads();
    uint32_t* mine = h[threadIdx.x >> 5];
    const unsigned long long n16 = n / 16;
    const uint4* v = reinterpret_cast<const uint4*>(sym);
    const bool aligned = ((uintptr_t) sym & 15) == 0;
    const unsigned long long stride = (unsigned long long) gridDim.x * blockDim.x;
    if (aligned) {
        for (unsigned long long i = (unsigned long long) blockIdx.x * blockDim.x + threadIdx.x;
             i < n16; i += stride) {
            const uint4 q = __ldg(v + i);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int t = 0; t < 16; ++t) atomicAdd(&mine[(w[t >> 2] >> (8 * (t & 3))) & 0xffu], 1u);
        }
    }
    for (unsigned long long i = (aligned ? n16 * 16 : 0) + (unsigned long long) blockIdx.x * blockDim.x +
                                threadIdx.x;
         i < n; i += stride)
        atomicAdd(&mine[sym[i]], 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < 256; b += blockDim.x) {
        uint32_t c = 0;
        for (int w = 0; w < 8; ++w) c += h[w][b];
        if (c) atomicAdd(hist + b, (unsigned long long) c);
    }
}

struct EncLayout {
    size_t status, result, end, ctr, tile_map, tile_sum, key, zero_end, node, start, total;
};

size_t al256(size_t x) { return (x + 255) & ~(size_t) 255; }

struct EncPlan {
    uint32_t Bs, nb, D, nblk, nseed;
};

EncLayout enc_layout(const EncPlan& e) {
    EncLayout a;
    size_t o = 0;
    const size_t ntiles = ((size_t) e.nblk + kLatScanTile - 1) / kLatScanTile;
    a.status = o; o += 256;
    a.result = o; o += 256;
    a.end = o; o += 256;
    a.ctr = o; o += 256;
    a.tile_map = o; o += al256(ntiles * 8);
    a.tile_sum = o; o += al256(ntiles * 8);
    a.key = o; o += al256((size_t) e.nblk * e.D * 4);
    a.zero_end = o;
    a.node = o; o += al256((size_t) e.nblk * e.D * 4);
    a.start = o; o += al256((size_t) e.nblk * 8);
    a.total = o;
    return a;
}

// Blocks of 128 bytes (64 on short inputs with small tables, whose encodes
// meet within a few hundred bytes), and starts every `hint` bytes or as many
// as run side by side (32 warps on every SM; 64 MB: 16 warps 414 us, 32 371),
// but no closer than the slots allow: every L / 12 bytes keeps up to 15
// distinct trajectories under way for the generator's data from 3.8 to 0.07
// bits per symbol (CPU simulation: L = 4096, 0.67 bits, 16 at 341 bytes).
// 1 MB at 1.5 bits, L = 4096: every 512 bytes 488 us, every 256 bytes 330.
EncPlan enc_plan(unsigned long long n, uint32_t L, uint32_t hint) {
    EncPlan e;
    e.Bs = n <= kEncSmallBytes && L <= 1024 ? 64 : 128;
    e.D = kEncSlots;
    const unsigned long long nblk = (n + e.Bs - 1) / e.Bs;
    const unsigned long long par = n / (152ull * 32 * 32);
    unsigned long long s = hint ? hint : std::max<unsigned long long>({par, L / 12, 128});
    s = std::min<unsigned long long>(std::max<unsigned long long>(s / e.Bs, 1), 1u << 28);
    e.nb = (uint32_t) s;
    e.nblk = (uint32_t) std::min<unsigned long long>(nblk, 0xffffffffull);
    e.nseed = (uint32_t) ((nblk + s - 1) / s);
    return e;
}

size_t enc_sync_smem(uint32_t L, uint32_t Bs, uint32_t threads) {
    return enc_table_bytes(L) + (size_t) threads * enc_pair_bytes(Bs);
}

size_t enc_final_smem(uint32_t L, uint32_t Bs, uint32_t threads) {
    uint32_t lg = 0;
    while ((1u << lg) < L) ++lg;
    return enc_table_bytes(L) +
           (size_t) (threads / 32) * (32 * enc_row_bytes(Bs) + enc_stage_words(Bs, lg) * 4);
}

int enc_sms() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1);
}

// Opts the kernels in to large dynamic shared memory, once per device.
void enc_attributes() {
    static std::mutex mu;
    static uint64_t done = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 64 && ((done >> dev) & 1)) return;
    cudaFuncSetAttribute(k_enc_sync<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    cudaFuncSetAttribute(k_enc_sync<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    cudaFuncSetAttribute(k_enc_final<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    cudaFuncSetAttribute(k_enc_final<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    if (dev < 64) done |= 1ull << dev;
}

}  // namespace
}  // namespace mans

using namespace mans;

extern "C" {

size_t mans_encode_blob_words(uint32_t L) { return 512 + (size_t) (L + 1) / 2; }

size_t mans_encode_max_units(size_t n, uint32_t L) {
    uint32_t lg = 0;
    while ((1u << lg) < L && lg < 31) ++lg;
    return (size_t) ((n * (unsigned long long) lg) / 32) + 6;
}

size_t mans_encode_aux_size(size_t n, uint32_t chunk_hint) {
    if (n == 0) return 0;
    return enc_layout(enc_plan(n, 2, chunk_hint)).total;   // the smallest blocks
}

int mans_encode(const uint8_t* d_sym, size_t n, const uint32_t* d_enc_blob, uint32_t L,
                uint32_t* d_units, size_t cap_units, void* d_aux, size_t aux_bytes,
                uint32_t chunk_hint, void* stream) {
    if (!d_sym || !d_enc_blob || !d_units || !d_aux || n == 0 || L < 2 || L > 8192 ||
        (L & (L - 1)) != 0 || ((uintptr_t) d_sym & 15) != 0 || ((uintptr_t) d_enc_blob & 3) != 0)
        return MANS_ERR_ARG;
    const EncPlan e = enc_plan(n, L, chunk_hint);
    if (e.nblk > 0xfffff000u) return MANS_ERR_ARG;   // 549 GB
    const EncLayout lay = enc_layout(e);
    if (aux_bytes < lay.total) return MANS_ERR_AUX_SMALL;
    if (cap_units < mans_encode_max_units(n, L)) return MANS_ERR_AUX_SMALL;
    cudaStream_t st = (cudaStream_t) stream;
    char* base = (char*) d_aux;
    EncParams p;
    std::memset(&p, 0, sizeof(p));
    p.sym = d_sym;
    p.n = n;
    p.blob = d_enc_blob;
    p.L = L;
    p.Bs = e.Bs;
    p.nb = e.nb;
    p.D = e.D;
    p.nblk = e.nblk;
    p.nseed = e.nseed;
    p.key = (uint32_t*) (base + lay.key);
    p.node = (uint32_t*) (base + lay.node);
    p.start = (unsigned long long*) (base + lay.start);
    p.tile_map = (unsigned long long*) (base + lay.tile_map);
    p.tile_sum = (unsigned long long*) (base + lay.tile_sum);
    p.ctr = (uint32_t*) (base + lay.ctr);
    p.status = (uint32_t*) (base + lay.status);
    p.result = (EncResult*) (base + lay.result);
    p.end = (EncEnd*) (base + lay.end);
    p.units = d_units;
    p.cap = cap_units;
    enc_attributes();
    const uint32_t sms = (uint32_t) enc_sms();
    const size_t words = lay.zero_end / 16 + cap_units / 4;
    const unsigned gz = (unsigned) std::min<size_t>((words + 1023) / 1024, 4 * sms);
    k_enc_zero<<<gz, 256, 0, st>>>((uint4*) base, lay.zero_end / 16, d_units, cap_units);
    const bool early = e.nseed <= 64 * sms;   // narrow warps below
    {
        // few trajectories: narrow warps spread over the schedulers of all SMs
        uint32_t th = kEncThreads;
        p.width = e.nseed <= 32 * sms ? 8 : (e.nseed <= 64 * sms ? 16 : 32);
        if (e.nseed <= p.width * 4 * sms) th = 32;
        const uint32_t per_cta = (th / 32) * p.width;
        const unsigned grid = std::min<unsigned>((e.nseed + per_cta - 1) / per_cta,
                                                 sms * kEncCtas * (kEncThreads / th));
        const size_t sm = enc_sync_smem(L, e.Bs, th);
        launch_after(e.Bs == 64 ? k_enc_sync<64> : k_enc_sync<128>, grid, th, sm, st, early, p);
    }
    launch_after(k_enc_scan<kEncSlots>, (e.nblk + kLatScanTile - 1) / kLatScanTile, kLatScanThreads,
                 lat_scan_smem(mans_encode_blob_words(L)), st, early, p);
    {
        const unsigned groups = (e.nblk + 31) / 32;
        uint32_t th = kEncFinalThreads;
        while (th > 64 && groups < (th / 32) * 2u * sms) th /= 2;
        const size_t sm = enc_final_smem(L, e.Bs, th);
        auto* k = e.Bs == 64 ? k_enc_final<64> : k_enc_final<128>;
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, th, sm) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        const unsigned need = (groups + th / 32 - 1) / (th / 32);
        launch_after(k, std::min<unsigned>(need, (unsigned) per_sm * sms), th, sm, st, early, p);
    }
    return cudaGetLastError() == cudaSuccess ? MANS_OK : MANS_ERR_CUDA;
}

int mans_encode_result(const void* d_aux, void* stream, uint64_t* n_units, uint32_t* first_bit,
                       uint32_t* first_state, uint32_t* dev_status) {
    if (!d_aux) return MANS_ERR_ARG;
    cudaStream_t st = (cudaStream_t) stream;
    uint32_t status = 0;
    EncResult r;
    const char* base = (const char*) d_aux;
    if (cudaMemcpyAsync(&status, base, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaMemcpyAsync(&r, base + 256, sizeof(r), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return MANS_ERR_CUDA;
    if (dev_status) *dev_status = status;
    if (n_units) *n_units = r.n_units;
    if (first_bit) *first_bit = r.first_bit;
    if (first_state) *first_state = r.first_state;
    if (status & MANS_DEV_SYNC_OVERFLOW) return MANS_ERR_SYNC;
    if (status & (MANS_DEV_SCAN_TIMEOUT)) return MANS_ERR_CUDA;
    if (status & MANS_DEV_COUNT_MISMATCH) return MANS_ERR_AUX_SMALL;
    return MANS_OK;
}

int mans_encode_sync(const uint8_t* d_sym, size_t n, const uint32_t* d_enc_blob, uint32_t L,
                     uint32_t* d_units, size_t cap_units, void* d_aux, size_t aux_bytes,
                     void* stream, uint64_t* n_units, uint32_t* first_bit,
                     uint32_t* first_state) {
    // a true path that ran out of slots: starts four times as far apart, in
    // the same workspace, until one trajectory encodes everything
    uint32_t chunk = 0;
    for (int attempt = 0; attempt < 8; ++attempt) {
        int rc = mans_encode(d_sym, n, d_enc_blob, L, d_units, cap_units, d_aux, aux_bytes, chunk,
                             stream);
        if (rc != MANS_OK) return rc;
        uint32_t dev = 0;
        rc = mans_encode_result(d_aux, stream, n_units, first_bit, first_state, &dev);
        if (rc != MANS_ERR_SYNC) return rc;
        const EncPlan e = enc_plan(n, L, chunk);
        if (e.nseed <= 1) return rc;
        chunk = (uint32_t) std::min<uint64_t>((uint64_t) e.nb * e.Bs * 4, 1u << 30);
    }
    return MANS_ERR_SYNC;
}

int mans_histogram(const uint8_t* d_sym, size_t n, uint64_t* d_hist, void* stream) {
    if (!d_sym || !d_hist) return MANS_ERR_ARG;
    cudaStream_t st = (cudaStream_t) stream;
    if (cudaMemsetAsync(d_hist, 0, 256 * sizeof(uint64_t), st) != cudaSuccess) return MANS_ERR_CUDA;
    if (n == 0) return MANS_OK;
    const unsigned grid = (unsigned) std::min<size_t>((n + kHistBytes - 1) / kHistBytes, 152 * 8);
    k_hist<<<grid, 256, 0, st>>>(d_sym, n, (unsigned long long*) d_hist);
    return cudaGetLastError() == cudaSuccess ? MANS_OK : MANS_ERR_CUDA;
}

}  // extern "C"
