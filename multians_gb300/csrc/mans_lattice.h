// Host interface of the lattice decode (mans_lattice.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace mans {

struct LatPlan {
    uint32_t B;       // units per block
    uint32_t nb;      // blocks between starts
    uint32_t D;       // slots per block
    uint32_t nblk;
    uint32_t nseed;
    uint32_t L;
    size_t bytes;     // workspace
};

// The geometry of a lattice decode of n_units units in at most `bytes` of
// workspace; `meet` is the mean meeting distance in units and `lanes` the
// trajectories the GPU runs side by side for this stream.  False when no
// geometry fits.
bool lat_plan(size_t n_units, size_t n_out, uint32_t L, double meet, uint32_t lanes, size_t bytes,
              LatPlan* out);

// A short stream leaves the GPU idle and takes as long as its longest
// trajectory, which ends sooner the more others it can meet: the geometry
// with 32 slots a block and starts closer by a quarter at least, on up to 512
// scan tiles.  False when
// there is none in `bytes`.  For streams whose chain is longer than the work
// of everything that runs beside it (lat_cost): sync pass of 146 KB at 3.1
// bits per symbol, L = 4096: 290 -> 132 us, of 5 MB at 2.5 576 -> 308; on all
// streams of a batch of 256 MB 584 -> 633.
bool lat_deep(size_t n_units, size_t n_out, uint32_t L, double meet, size_t bytes,
              const LatPlan& base, LatPlan* out);

// Sync pass of a plan, estimated: its longest chain (24 ns a step), and its
// steps at the rate of a full GPU (1 M a microsecond).
struct LatCost {
    double chain_us, work_us;
};
LatCost lat_cost(size_t n_units, size_t n_out, double meet, const LatPlan& plan);

// Workspace of a lattice of nblk blocks with 16 slots each; a plan uses what
// it is given, 32 slots a block where they fit.
size_t lat_bytes(size_t nblk);

struct LatCall {
    const uint32_t* units;
    size_t n_units;
    uint8_t* out;
    size_t n_out;
    const uint32_t* table;
    uint32_t L, first_idx, first_pos, flags;
};

// Enqueues the decode in the workspace at d_aux (its first word is the
// status).  `mark(i)` is called before each of the five timed kernel slots
// and after the last.  Returns the number of kernels, or 0 on a CUDA error.
uint32_t lat_decode(const LatCall& call, const LatPlan& plan, void* d_aux, cudaStream_t stream,
                    void (*mark)(int, cudaStream_t));

// What the trajectories of the last lattice decode in d_aux cost (waits for
// the stream): blocks decoded by all of them, blocks of the longest.
bool lat_stats(const void* d_aux, cudaStream_t stream, uint64_t* visits, uint64_t* longest);

// Batched decodes.  The parameters of a stream are lat_params_size() bytes;
// the batch keeps one array of them and lists of work items on the device.
struct LatItem {
    uint32_t stream;
    uint32_t index;
    uint32_t count;
    uint32_t pad;
};
struct LatSmem {
    size_t prep, sync, scan, final;
};
constexpr uint32_t kLatBatchWarps = 4;   // of a sync-pass CTA

// Lanes of a sync-pass warp that run trajectories: narrow warps while 16 of
// them an SM hold every start.
uint32_t lat_width(uint64_t starts, uint32_t sms);

size_t lat_params_size();
void lat_fill_params(void* dst, const LatCall& call, const LatPlan& plan, void* slice,
                     uint32_t* d_status, uint32_t width);
uint32_t lat_prep_items(const LatPlan& plan);
uint32_t lat_scan_tiles(const LatPlan& plan);
uint32_t lat_final_ctas(const LatPlan& plan);
LatSmem lat_batch_smem(const LatCall& call, const LatPlan& plan);
void lat_batch_init();
void lat_batch_prep(const void* ps, const LatItem* items, size_t n, const LatSmem& sm,
                    cudaStream_t st);
void lat_batch_sync(const void* ps, const LatItem* items, size_t n, const LatSmem& sm,
                    uint32_t width, bool deep, cudaStream_t st);
void lat_batch_scan(const void* ps, const LatItem* items, size_t n, const LatSmem& sm,
                    bool deep, uint32_t* ticket, cudaStream_t st);
void lat_batch_final(const void* ps, const LatItem* items, size_t n, size_t smem, cudaStream_t st);

}  // namespace mans
