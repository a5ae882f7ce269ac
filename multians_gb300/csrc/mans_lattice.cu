// Lattice decode: kernels and launches (the method is in mans_lattice.cuh).
#include "mans_lattice.h"

#include <algorithm>
#include <cmath>
#include <mutex>

#include "mans_lattice.cuh"

namespace mans {
namespace {

constexpr uint32_t kLatPrepThreads = 1024;
constexpr size_t kLatZeroBytes = 128 * 1024;   // zeroed by a CTA

// Tables (first CTA) and the zeroed words: counters, look-back words, slots.
__global__ void __launch_bounds__(kLatPrepThreads) k_lat_prep(LatParams p, uint4* zero, size_t n16) {
    follow_previous();
    if (blockIdx.x == 0) lat_tables(p);
    const size_t stride = (size_t) gridDim.x * blockDim.x;
    for (size_t i = (size_t) blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride)
        zero[i] = make_uint4(0, 0, 0, 0);
}

// Groups of four slots of the next block that a trajectory looks at ahead.
constexpr uint32_t lat_ahead(uint32_t D, bool narrow) { return D > 16 ? 4 : (narrow ? 2 : 1); }

template <uint32_t kB, bool kNarrow, uint32_t kV>
__global__ void __launch_bounds__(kLatThreads) k_lat_sync(LatParams p) {
    follow_previous();
    lat_sync_body<kB, kNarrow, kV>(p, p.ctr + kLatNext, p.nseed);
}

template <uint32_t kD>
__global__ void __launch_bounds__(kLatScanThreads, kD > 16 ? 2 : 5) k_lat_scan(LatParams p) {
    __shared__ uint32_t s_tile;
    follow_previous();
    if (threadIdx.x == 0) s_tile = atomicAdd(p.ctr + kLatTicket, 1u);
    __syncthreads();
    lat_scan_body<LatParams, kD>(p, s_tile);
}

template <bool kRev, uint32_t kB>
__global__ void __launch_bounds__(kLatFinalThreads) k_lat_final(LatParams p) {
    follow_previous();
    lat_final_body<kRev, kB>(p, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------------------
// Batches: every CTA takes one work item {stream, index, count} of a
// host-built list and its stream's parameters.

__device__ __forceinline__ void lat_load_params(LatParams& dst, const LatParams* src) {
    static_assert(sizeof(LatParams) % 4 == 0, "word copy");
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
    for (uint32_t i = threadIdx.x; i < sizeof(LatParams) / 4; i += blockDim.x) d[i] = s[i];
    __syncthreads();
}

// index 0 builds the stream's tables; the others zero a share of its words
// from the counters to the end of the slots.
__global__ void __launch_bounds__(kLatPrepThreads) k_lat_prep_batch(const LatParams* ps,
                                                                    const LatItem* items) {
    __shared__ LatParams sp;
    const LatItem it = items[blockIdx.x];
    lat_load_params(sp, ps + it.stream);
    if (it.index == 0) {
        lat_tables(sp);
        return;
    }
    uint4* z = reinterpret_cast<uint4*>(sp.ctr);
    const size_t n16 = ((char*) sp.tab_cnt - (char*) sp.ctr) / 16;
    const size_t stride = (size_t) (it.count - 1) * blockDim.x;
    for (size_t i = (size_t) (it.index - 1) * blockDim.x + threadIdx.x; i < n16; i += stride)
        z[i] = make_uint4(0, 0, 0, 0);
}

template <bool kNarrow, uint32_t kV>
__device__ __forceinline__ void lat_sync_any(const LatParams& p, uint32_t* next, uint32_t limit) {
    if (p.B == 4) lat_sync_body<4, kNarrow, kV>(p, next, limit);
    else if (p.B == 8) lat_sync_body<8, kNarrow, kV>(p, next, limit);
    else if (p.B == 16) lat_sync_body<16, kNarrow, kV>(p, next, limit);
    else lat_sync_body<32, kNarrow, kV>(p, next, limit);
}

// index: the CTA's first start, count: the end of its starts.
template <bool kNarrow, bool kDeep>
__global__ void __launch_bounds__(kLatThreads) k_lat_sync_batch(const LatParams* ps,
                                                                const LatItem* items) {
    __shared__ LatParams sp;
    __shared__ uint32_t s_next;
    const LatItem it = items[blockIdx.x];
    if (threadIdx.x == 0) s_next = it.index;
    lat_load_params(sp, ps + it.stream);
    if (kDeep && sp.D > 16) lat_sync_any<kNarrow, lat_ahead(32, kNarrow)>(sp, &s_next, it.count);
    else lat_sync_any<kNarrow, lat_ahead(16, kNarrow)>(sp, &s_next, it.count);
}

// The ticket hands items out in list order, which holds each stream's tiles
// in increasing order: a tile only waits on tiles that have started.
template <bool kDeep>
__global__ void __launch_bounds__(kLatScanThreads) k_lat_scan_batch(const LatParams* ps,
                                                                    const LatItem* items,
                                                                    uint32_t* ticket) {
    __shared__ LatParams sp;
    __shared__ uint32_t s_item;
    if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1u);
    __syncthreads();
    const LatItem it = items[s_item];
    lat_load_params(sp, ps + it.stream);
    if (kDeep && sp.D == 32) lat_scan_body<LatParams, 32>(sp, it.index);
    else if (sp.D == 4) lat_scan_body<LatParams, 4>(sp, it.index);
    else if (sp.D == 8) lat_scan_body<LatParams, 8>(sp, it.index);
    else if (sp.D == 12) lat_scan_body<LatParams, 12>(sp, it.index);
    else lat_scan_body<LatParams, 16>(sp, it.index);
}

template <bool kRev>
__device__ __forceinline__ void lat_final_any(const LatParams& p, const LatItem& it) {
    if (p.B == 4) lat_final_body<kRev, 4>(p, it.index, it.count);
    else if (p.B == 8) lat_final_body<kRev, 8>(p, it.index, it.count);
    else if (p.B == 16) lat_final_body<kRev, 16>(p, it.index, it.count);
    else lat_final_body<kRev, 32>(p, it.index, it.count);
}

// index: the CTA of the stream's count.
__global__ void __launch_bounds__(kLatFinalThreads) k_lat_final_batch(const LatParams* ps,
                                                                      const LatItem* items) {
    __shared__ LatParams sp;
    const LatItem it = items[blockIdx.x];
    lat_load_params(sp, ps + it.stream);
    if (sp.flags & MANS_DECODE_SOURCE_ORDER) lat_final_any<true>(sp, it);
    else lat_final_any<false>(sp, it);
}

static_assert(kLatThreads == 32 * kLatBatchWarps, "batch items");

// CTAs of kLatThreads a persistent sync pass keeps on an SM: 16 warps, near
// the rate its shared-memory lookups allow.
constexpr uint32_t kLatCtas = 4;

size_t align256(size_t x) { return (x + 255) & ~(size_t) 255; }

struct LatLayout {
    size_t ctr, tile_map, tile_sum, key, zero_end, tab_cnt, tab_sym, node, start, total;
};

LatLayout lat_layout(size_t nblk, uint32_t D, uint32_t L) {
    LatLayout a;
    const size_t ntiles = (nblk + kLatScanTile - 1) / kLatScanTile;
    size_t o = 256;   // status
    a.ctr = o; o += 256;
    a.tile_map = o; o += align256(ntiles * 8);
    a.tile_sum = o; o += align256(ntiles * 8);
    a.key = o; o += align256(nblk * D * 4);
    a.zero_end = o;
    a.tab_cnt = o; o += align256((size_t) L * 4);
    a.tab_sym = o; o += align256((size_t) L * 4);
    a.node = o; o += align256(nblk * D * 4);
    a.start = o; o += align256(nblk * 8);
    a.total = o;
    return a;
}

size_t lat_sync_smem(uint32_t L, uint32_t B, uint32_t threads) {
    return (((size_t) L * 4 + 15) & ~(size_t) 15) + lat_ring_bytes(B) * (threads / 32);
}

constexpr size_t kLatFinalSmemMax = 200 * 1024;
size_t lat_final_smem(uint32_t L, uint32_t B, uint32_t stage_cap, uint32_t threads) {
    return (((size_t) L * 4 + 15) & ~(size_t) 15) +
           (size_t) (threads / 32) * (lat_final_warp_bytes(B) + stage_cap + 16);
}

// Staging bytes per warp of the final pass: 1.25x the expected symbols of
// 32 blocks, as far as eight warps fit an SM's shared memory.
uint32_t lat_stage_cap(double per_unit, uint32_t B, uint32_t L) {
    uint64_t cap = (uint64_t) (per_unit * 32.0 * B * 1.25) + 128;
    cap = std::min<uint64_t>(std::max<uint64_t>(cap, 512), 16384);
    const size_t warps = kLatFinalThreads / 32;
    const size_t room = (kLatFinalSmemMax - lat_final_smem(L, B, 0, kLatFinalThreads)) / warps;
    cap = std::min<uint64_t>(cap, room & ~(size_t) 15);
    return (uint32_t) ((cap + 15) & ~(uint64_t) 15);
}

int sm_count() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(sms, 1);
}

template <bool kNarrow, uint32_t kD>
void (*sync_kernel(uint32_t B))(LatParams) {
    constexpr uint32_t kV = lat_ahead(kD, kNarrow);
    return B == 4 ? k_lat_sync<4, kNarrow, kV>
                  : (B == 8 ? k_lat_sync<8, kNarrow, kV>
                            : (B == 16 ? k_lat_sync<16, kNarrow, kV> : k_lat_sync<32, kNarrow, kV>));
}
void (*sync_kernel(uint32_t B, uint32_t D, bool narrow))(LatParams) {
    return D > 16 ? (narrow ? sync_kernel<true, 32>(B) : sync_kernel<false, 32>(B))
                  : (narrow ? sync_kernel<true, 16>(B) : sync_kernel<false, 16>(B));
}

auto batch_sync(bool narrow, bool deep) {
    return narrow ? (deep ? k_lat_sync_batch<true, true> : k_lat_sync_batch<true, false>)
                  : (deep ? k_lat_sync_batch<false, true> : k_lat_sync_batch<false, false>);
}

// Opts the kernels in to large dynamic shared memory, once per device.
void lat_attributes() {
    static std::mutex mu;
    static uint64_t done = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 64 && ((done >> dev) & 1)) return;
    const auto set = [](auto* k) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int) kLatFinalSmemMax);
    };
    set(k_lat_prep); set(k_lat_prep_batch); set(k_lat_final_batch);
    set(batch_sync(false, false)); set(batch_sync(false, true));
    set(batch_sync(true, false)); set(batch_sync(true, true));
    for (uint32_t B = 4; B <= 32; B *= 2)
        for (uint32_t D = 16; D <= 32; D *= 2) {
            set(sync_kernel(B, D, false));
            set(sync_kernel(B, D, true));
        }
    set(k_lat_final<false, 4>); set(k_lat_final<false, 8>); set(k_lat_final<false, 16>);
    set(k_lat_final<false, 32>); set(k_lat_final<true, 32>);
    set(k_lat_final<true, 4>); set(k_lat_final<true, 8>); set(k_lat_final<true, 16>);
    if (dev < 64) done |= 1ull << dev;
}

template <bool kRev>
void (*final_kernel(uint32_t B))(LatParams) {
    return B == 4 ? k_lat_final<kRev, 4>
                  : (B == 8 ? k_lat_final<kRev, 8>
                            : (B == 16 ? k_lat_final<kRev, 16> : k_lat_final<kRev, 32>));
}

LatParams lat_params(const LatCall& call, const LatPlan& plan, char* base) {
    const LatLayout a = lat_layout(plan.nblk, plan.D, call.L);
    LatParams p{};
    p.units = call.units;
    p.out = call.out;
    p.table = call.table;
    p.status = (uint32_t*) base;
    p.ctr = (uint32_t*) (base + a.ctr);
    p.tile_map = (unsigned long long*) (base + a.tile_map);
    p.tile_sum = (unsigned long long*) (base + a.tile_sum);
    p.key = (uint32_t*) (base + a.key);
    p.tab_cnt = (uint32_t*) (base + a.tab_cnt);
    p.tab_sym = (uint32_t*) (base + a.tab_sym);
    p.node = (uint32_t*) (base + a.node);
    p.start = (unsigned long long*) (base + a.start);
    p.n_out = call.n_out;
    p.n_units = (uint32_t) call.n_units;
    p.L = call.L;
    p.first_idx = call.first_idx;
    p.first_pos = call.first_pos;
    p.B = plan.B;
    p.nb = plan.nb;
    p.D = plan.D;
    p.nblk = plan.nblk;
    p.nseed = plan.nseed;
    p.stage_cap = lat_stage_cap((double) call.n_out / (double) call.n_units, plan.B, call.L);
    p.flags = call.flags;
    return p;
}

}  // namespace

uint32_t lat_width(uint64_t starts, uint32_t sms) {
    // A warp waits for the slowest of its trajectories at every block, so with
    // few of them each gets a warp (219 KB at 0.7 bits per symbol, L = 4096: 8
    // lanes 277 us, 1 lane 253), and the CTA's barrier goes (48 streams: 400
    // -> 393 us).  Past 16 warps an SM wider ones are as fast (16 lanes: 1.2
    // MB 52 us either way).
    uint32_t w = 1;
    while (w <= 8 && starts > w * 16ull * sms) w *= 2;
    return w <= 8 ? w : 32;
}

size_t lat_bytes(size_t nblk) { return lat_layout(nblk, 16, kMaxStates).total; }

// Blocks and starts for starts every `s` units (s_par: the distance at which
// they fill the lanes) and D slots.
static bool lat_fit(size_t n_units, size_t n_out, uint32_t L, double s, double s_par, uint32_t D,
                    size_t bytes, LatPlan* o) {
    // About 128 symbols per block: the final pass stages 32 blocks a warp, and
    // a step's share of a block's bookkeeping stays below a tenth.  Blocks of
    // 32 units from 5.3 bits per symbol on (256 MB at 6 bits: 691 -> 629 us,
    // 512 MB at 8.6 bits 1511 -> 1192, the scan and the slots' traffic halved).
    const double spu = (double) n_out / (double) n_units;
    uint32_t B = 32;
    while (B > 4 && spu * B > 192.0) B /= 2;
    while (B > 4 && B > s && spu * B >= 96.0) B /= 2;
    for (; B <= 32; B *= 2) {
        const size_t nblk = n_units / B + 1;
        if (nblk * D > 0xffffffffull) continue;
        const size_t need = lat_layout(nblk, D, L).total;
        if (need > bytes) continue;
        o->B = B;
        // rounded up, so that starts never outnumber the lanes of one wave
        o->nb = (uint32_t) std::max(1.0, s > s_par ? std::floor(s / B + 0.5) : std::ceil(s / B));
        o->D = D;
        o->nblk = (uint32_t) nblk;
        o->nseed = (uint32_t) ((nblk + o->nb - 1) / o->nb);
        o->L = L;
        o->bytes = need;
        return true;
    }
    return false;
}

// Starts every s units: as many as run side by side, but no closer than the
// slots allow.  About 1.2 sqrt(2 T / s) distinct trajectories are under way at
// a place on average, and twice that at most over a long stream: s = meet /
// kPerMeet[D / 4 - 1] leaves room for a T 2.7 times the model's (symbols of
// equal frequency meet that late).  Closer ones run out of slots: 3 M of eight
// equally frequent symbols, L = 1024, 12 slots, s = meet / 4: 3 blocks
// repaired, 0.6 ms; meet / 8: 5812 blocks, 86 ms.
static constexpr double kPerMeet[4] = {0.17, 1.0, 4.0, 6.8};
static constexpr double kPerMeetDeep = 29.0;   // 32 slots
static constexpr double kMinSpacing = 4.0;     // units
// Scan tiles of a lattice with 32 slots: one tile hands its end to the next in
// order, 0.5 us each, where with fewer slots the maps are composed ahead.  A
// stream of 2 bits per symbol, L = 1024, beside twelve sparse ones: 352 tiles
// 2499 us (with 16 slots 2697), 880 tiles 5849 (5414), 3553 tiles 22.4 ms (19.2).
static constexpr uint32_t kDeepTiles = 512;

bool lat_plan(size_t n_units, size_t n_out, uint32_t L, double meet, uint32_t lanes, size_t bytes,
              LatPlan* out) {
    if (n_out >> (63 - kLatEntBits)) return false;
    const double s_par = std::max((double) n_units / lanes, kMinSpacing);
    // Codes of nearly one length: trajectories at different bit phases meet at
    // the rare other codes only, however short the mean distance of a table of
    // a few states is.  With four slots 16 MB at 3.98 bits, L = 16, need 973
    // blocks repaired (8.1 ms), with eight none (134 us).  From L = 64 on four
    // did at every size and compression tried, and eight cost 5 to 10 %.
    const bool phases = L <= 32 && 32.0 * n_units >= 0.95 * std::log2((double) L) * n_out;
    uint32_t D = phases ? 8 : 4;
    while (D < 16 && s_par < meet / kPerMeet[D / 4 - 1]) D += 4;
    for (; D >= 4; D -= 4)
        if (lat_fit(n_units, n_out, L, std::max(s_par, meet / kPerMeet[D / 4 - 1]), s_par, D, bytes,
                    out))
            return true;
    return false;
}

bool lat_deep(size_t n_units, size_t n_out, uint32_t L, double meet, size_t bytes,
              const LatPlan& base, LatPlan* out) {
    // shorter blocks gain nothing (128 KB at 3.8 bits, L = 1024, blocks of 16
    // -> 8: 67 us both, and 6 us more in the scan)
    const double s = std::max(meet / kPerMeetDeep, kMinSpacing);
    return lat_fit(n_units, n_out, L, s, kMinSpacing, 32, bytes, out) && out->B >= base.B &&
           4ull * out->nb * out->B <= 3ull * base.nb * base.B &&
           lat_scan_tiles(*out) <= kDeepTiles;
}

LatCost lat_cost(size_t n_units, size_t n_out, double meet, const LatPlan& plan) {
    // a trajectory meets one of the m - 1 others at its place; the longest
    // of a stream goes about four times as far as the mean (simulated)
    const double s = (double) plan.nb * plan.B;
    const double m = std::max(1.0, 1.2 * std::sqrt(2.0 * meet / s));
    // zero-bit steps are folded: two bits a step at least
    const double steps = std::min(n_out / (double) n_units, 15.5);
    return {std::min(4.0 * m * s, (double) n_units) * steps * 0.024, n_units * m * steps * 1e-6};
}

uint32_t lat_decode(const LatCall& call, const LatPlan& plan, void* d_aux, cudaStream_t st,
                    void (*mark)(int, cudaStream_t)) {
    char* base = (char*) d_aux;
    const LatLayout a = lat_layout(plan.nblk, plan.D, call.L);
    LatParams p = lat_params(call, plan, base);
    lat_attributes();
    const int sms = sm_count();
    const size_t n16 = (a.zero_end - a.ctr) / 16;
    mark(0, st);
    const unsigned gz = 1 + (unsigned) std::min<size_t>((n16 * 16 + kLatZeroBytes - 1) / kLatZeroBytes,
                                                        2 * sms - 1);
    k_lat_prep<<<gz, kLatPrepThreads, (size_t) call.L * 12, st>>>(p, (uint4*) (base + a.ctr), n16);
    mark(1, st);
    const uint32_t width = lat_width(plan.nseed, sms);
    // short: the sync pass leaves room beside it (4 KB 75 -> 67 us; where it
    // fills the GPU waiting CTAs cost more: 256 MB 541 -> 582, 16 MB 178 -> 185)
    const bool early = width < 32;
    // sync pass
    {
        const uint32_t th = plan.nseed <= width * 4 * sms ? 32 : kLatThreads;
        p.width = width;
        const unsigned need = (plan.nseed + (th / 32) * width - 1) / ((th / 32) * width);
        const unsigned grid = std::min<unsigned>(need, (unsigned) sms * kLatCtas * (kLatThreads / th));
        const size_t sm = lat_sync_smem(call.L, plan.B, th);
        launch_after(sync_kernel(plan.B, plan.D, width < 32), grid, th, sm, st, early, p);
    }
    mark(2, st);
    mark(3, st);
    {
        const unsigned g = (plan.nblk + kLatScanTile - 1) / kLatScanTile;
        const size_t sm = lat_scan_smem(call.L);
        auto* k = plan.D == 4    ? k_lat_scan<4>
                  : plan.D == 8  ? k_lat_scan<8>
                  : plan.D == 12 ? k_lat_scan<12>
                  : plan.D == 16 ? k_lat_scan<16>
                                 : k_lat_scan<32>;
        launch_after(k, g, kLatScanThreads, sm, st, early, p);
    }
    mark(4, st);
    {
        const unsigned groups = (plan.nblk + 31) / 32;
        uint32_t th = kLatFinalThreads;
        while (th > 64 && groups < (th / 32) * 2u * sms) th /= 2;
        const size_t sm = lat_final_smem(call.L, plan.B, p.stage_cap, th);
        auto* k = (call.flags & MANS_DECODE_SOURCE_ORDER) ? final_kernel<true>(plan.B)
                                                          : final_kernel<false>(plan.B);
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, th, sm) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        const unsigned need = (groups + th / 32 - 1) / (th / 32);
        launch_after(k, std::min<unsigned>(need, (unsigned) (per_sm * sms)), th, sm, st, early, p);
    }
    mark(5, st);
    return cudaGetLastError() == cudaSuccess ? 4u : 0u;
}

bool lat_stats(const void* d_aux, cudaStream_t st, uint64_t* visits, uint64_t* longest) {
    uint32_t c[8] = {};
    if (cudaMemcpyAsync(c, (const char*) d_aux + 256, sizeof(c), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return false;
    *visits = c[kLatVisits];
    *longest = c[kLatMaxLife];
    return true;
}

size_t lat_params_size() { return sizeof(LatParams); }

void lat_fill_params(void* dst, const LatCall& call, const LatPlan& plan, void* slice,
                     uint32_t* d_status, uint32_t width) {
    LatParams p = lat_params(call, plan, (char*) slice);
    p.status = d_status;
    p.width = width;
    *(LatParams*) dst = p;
}

uint32_t lat_prep_items(const LatPlan& plan) {
    const LatLayout a = lat_layout(plan.nblk, plan.D, plan.L);
    return 1 + (uint32_t) ((a.zero_end - a.ctr + kLatZeroBytes - 1) / kLatZeroBytes);
}

uint32_t lat_scan_tiles(const LatPlan& plan) {
    return (plan.nblk + kLatScanTile - 1) / kLatScanTile;
}

uint32_t lat_final_ctas(const LatPlan& plan) {
    return (plan.nblk + kLatFinalThreads - 1) / kLatFinalThreads;
}

LatSmem lat_batch_smem(const LatCall& call, const LatPlan& plan) {
    LatSmem s;
    s.prep = (size_t) call.L * 12;
    s.sync = lat_sync_smem(call.L, plan.B, kLatThreads);
    s.scan = lat_scan_smem(call.L);
    s.final = lat_final_smem(
        call.L, plan.B, lat_stage_cap((double) call.n_out / (double) call.n_units, plan.B, call.L),
        kLatFinalThreads);
    return s;
}

void lat_batch_init() { lat_attributes(); }

void lat_batch_prep(const void* ps, const LatItem* items, size_t n, const LatSmem& sm,
                    cudaStream_t st) {
    if (n) k_lat_prep_batch<<<(unsigned) n, kLatPrepThreads, sm.prep, st>>>((const LatParams*) ps, items);
}
void lat_batch_sync(const void* ps, const LatItem* items, size_t n, const LatSmem& sm,
                    uint32_t width, bool deep, cudaStream_t st) {
    if (n) batch_sync(width < 32, deep)<<<(unsigned) n, kLatThreads, sm.sync, st>>>((const LatParams*) ps, items);
}
void lat_batch_scan(const void* ps, const LatItem* items, size_t n, const LatSmem& sm,
                    bool deep, uint32_t* ticket, cudaStream_t st) {
    auto* k = deep ? k_lat_scan_batch<true> : k_lat_scan_batch<false>;
    if (n) k<<<(unsigned) n, kLatScanThreads, sm.scan, st>>>((const LatParams*) ps, items, ticket);
}
void lat_batch_final(const void* ps, const LatItem* items, size_t n, size_t smem, cudaStream_t st) {
    if (n)
        k_lat_final_batch<<<(unsigned) n, kLatFinalThreads, smem, st>>>((const LatParams*) ps, items);
}

}  // namespace mans
