// Shared device helpers of the particle sort: key generation (cell id from
// float32 positions and Philox4x32-10 shuffle bits), small PTX wrappers and the
// workspace layout.  sm_100a only.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/aether_sort.h"

namespace aether {

constexpr int kShuffleBits = 7;  // radix_sort_reference.py:33
constexpr int kRadixBits = 8;    // digit width of this implementation
constexpr int kRadix = 1 << kRadixBits;
constexpr int kMaxPasses = 4;    // 32-bit keys / 8-bit digits

// Status word of the chained scan: flag in bits 30-31, count in bits 0-29.
// (The reference packs a 2-bit flag over a 29-bit count into a signed word,
// radix_sort_reference.py:36-40; the unsigned form here leaves 30 value bits.)
constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagInclusive = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kValueMask = ~kFlagMask;

// Error codes left in the workspace header by a device wait that gave up.
constexpr int kErrLookbackTimeout = 1;
constexpr int kErrBucketOverflow = 2;
constexpr int kErrBulkCopyTimeout = 3;
constexpr int kErrBarrierTimeout = 4;
constexpr int kErrReceiveOverflow = 5;
constexpr int kErrExchangeTimeout = 6;

constexpr int kMaxWorld = 8;    // ranks of the multi-GPU decomposition
constexpr int kMaxSlices = 32;  // slices of one rank's input in the sliced exchange

// What a rank receives in the sliced exchange, slice by slice (device memory, written by
// slab_exchange_prepare).  The received array is the concatenation over sources s of what s
// sent, in s's order; source s's slice k occupies [first[k][s], first[k][s] + length[k][s]).
// The local sort lays its records out with one chunk per slice: chunk k's records start at
// chunk_base[k] (the particles of all sources' slices before k).
struct SliceSegments {
  uint32_t n;        // particles received in all
  uint32_t slices;
  uint32_t sources;
  uint32_t pad;
  uint32_t chunk_base[kMaxSlices + 1];
  uint32_t first[kMaxSlices][kMaxWorld];
  uint32_t length[kMaxSlices][kMaxWorld];
};

constexpr int kMaxTiles = 512;  // tiles of the one-launch sort

// Workspace header (first 5 KiB of the workspace, zeroed by every call).
struct alignas(16) Header {
  int32_t error;              // first error code seen, 0 when clean
  int32_t use_standard;       // bucketed path: 1 when it handed over to the digit passes
  uint32_t phase_ticket, phase_done;  // run_phases: pieces handed out, pieces done
  uint32_t max_bucket;        // bucketed path: largest bucket seen
  uint32_t redo_groups;       // groups whose counters wrapped, to be finished bucket by bucket
  // One-launch sort: tiles counted and stored, next tile to look at for a block that helps,
  // groups cut, next task and tasks done of the finish.
  uint32_t tiles_counted, tiles_stored, help_next, groups, task_next, tasks_done;
  uint32_t settle_failed;     // the sort of a settled state gave the call to the general path
  uint32_t settle_large;      // buckets of the sort of a settled state that a block of its finish does not hold
  uint32_t settle_sampled;    // movers among the particles that its probe looked at
  uint32_t shared_rounds;     // rounds in which the count kernel has seen neighbours in one bucket
  uint32_t tile_claimed[kMaxTiles / 32], tile_loose[kMaxTiles / 32];  // one bit per tile
  uint32_t tile_counter[kMaxPasses];  // ticket dispenser of each digit pass
  uint32_t aux_counter[8];
  uint32_t pad[4];
  uint32_t digit_hist[kMaxPasses][kRadix];  // global digit histograms (upsweep)
};
// Bytes the hand-over to the digit passes does not clear: blocks that start late still look there.
constexpr size_t kHeaderKept = 192;
static_assert(offsetof(Header, tile_counter) == kHeaderKept && offsetof(Header, digit_hist) == 256, "header");
static_assert(sizeof(Header) % 256 == 0, "header must keep 256-byte alignment");

__host__ __device__ inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// Word 0 of Philox4x32-10 with counter (c0, 0, 0, 0) and key (k0, k1): the
// value tl.randint(seed, i) gives the reference's key kernel
// (fused_radix_sort.py:101), restated after the reference's own generator
// (cuda/philox.h:56-72).  The zero counter words let the first two rounds and
// the unused outputs of the last round fold away at compile time.
// One wide multiply gives both halves of a product (16 M particles sorted without
// payload: 373 -> 366 us per call against separate high and low multiplies).
__device__ __forceinline__ uint32_t philox_word0(uint32_t c0, uint32_t k0, uint32_t k1) {
  constexpr uint32_t kM0 = 0xD2511F53u, kM1 = 0xCD9E8D57u;
  constexpr uint32_t kW0 = 0x9E3779B9u, kW1 = 0xBB67AE85u;
  uint32_t c1 = 0, c2 = 0, c3 = 0;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    if (r > 0) {
      k0 += kW0;
      k1 += kW1;
    }
    const uint64_t p0 = static_cast<uint64_t>(kM0) * c0, p1 = static_cast<uint64_t>(kM1) * c2;
    const uint32_t hi0 = static_cast<uint32_t>(p0 >> 32), lo0 = static_cast<uint32_t>(p0);
    const uint32_t hi1 = static_cast<uint32_t>(p1 >> 32), lo1 = static_cast<uint32_t>(p1);
    c0 = hi1 ^ c1 ^ k0;
    c1 = lo1;
    c2 = hi0 ^ c3 ^ k1;
    c3 = lo0;
  }
  return c0;
}

// clamp(int32_rz((c - lo) * inv), 0, cells - 1) with separately rounded
// subtract and multiply (fused_radix_sort.py:93-98).  The intrinsics keep the
// compiler from contracting the pair into a fused multiply-add.
__device__ __forceinline__ int axis_index(float c, float lo, float inv, int cells) {
  const int i = __float2int_rz(__fmul_rn(__fsub_rn(c, lo), inv));
  return min(max(i, 0), cells - 1);
}

// Cell id over the x-slab [ix_offset, ix_offset + nx_local) of the grid.  A particle whose
// column lies outside the slab (the caller's precondition broken) is binned into the slab's
// nearest column: every table the kernels index with a cell id stays in range.
__device__ __forceinline__ uint32_t cell_of(float x, float y, float z, const AetherGrid& g) {
  const int ix = axis_index(x, g.x0, g.inv_dx, g.nx);
  const int iy = axis_index(y, g.y0, g.inv_dy, g.ny);
  const int iz = axis_index(z, g.z0, g.inv_dz, g.nz);
  const int ix_local = min(max(ix - g.ix_offset, 0), g.nx_local - 1);
  return static_cast<uint32_t>((iz * g.ny + iy) * g.nx_local + ix_local);
}

__device__ __forceinline__ uint32_t make_key(uint32_t cell, uint32_t index, uint32_t k0,
                                             uint32_t k1) {
  return (cell << kShuffleBits) | (philox_word0(index, k0, k1) >> (32 - kShuffleBits));
}

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Whether the call was handed over to the digit passes, one answer for the whole block (a
// barrier).  Other blocks may set the word while a kernel runs: threads that read it for
// themselves could disagree and meet different barriers.
__device__ __forceinline__ bool handed_over(const Header* hdr) {
  return __syncthreads_or(threadIdx.x == 0 &&
                          ld_relaxed(reinterpret_cast<const uint32_t*>(&hdr->use_standard)) != 0);
}
__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Adds one to a histogram bin per lane.  Lanes hitting the same bin share one add
// when the whole warp agrees, or (through match.any) when neighbouring lanes do.
__device__ __forceinline__ void bin_add(uint32_t* hist, uint32_t bin, bool valid) {
  const uint32_t active = __ballot_sync(0xffffffffu, valid);
  if (active == 0) return;
  const int first = __ffs(active) - 1;
  const uint32_t first_bin = __shfl_sync(0xffffffffu, bin, first);
  const bool uniform = __all_sync(0xffffffffu, !valid || bin == first_bin);
  if (uniform) {
    if (static_cast<int>(lane_id()) == first) atomicAdd(&hist[first_bin], __popc(active));
    return;
  }
  const uint32_t next_bin = __shfl_down_sync(0xffffffffu, bin, 1);
  const bool clustered = __any_sync(0xffffffffu, valid && lane_id() < 31 && next_bin == bin);
  if (clustered) {
    const uint32_t peers = __match_any_sync(0xffffffffu, valid ? bin : 0xffffffffu) & active;
    if (valid && (peers & lanemask_lt()) == 0) atomicAdd(&hist[bin], __popc(peers));
  } else if (valid) {
    atomicAdd(&hist[bin], 1u);
  }
}

// Exclusive scan of one value per thread over a block of up to 1024 threads;
// `warp_sum` is 32 words of shared memory, *total receives the block's sum.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sum,
                                                         uint32_t* total) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < static_cast<int>((blockDim.x + 31) >> 5) ? warp_sum[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    warp_sum[lane] = wi - w;
    if (lane == 31) *total = wi;
  }
  __syncthreads();
  return warp_sum[warp] + incl - v;
}

// Streaming (read-once / write-once) accesses: keep them from displacing data
// that is reused out of L2.
__device__ __forceinline__ float4 ldcs4(const float* p) {
  return __ldcs(reinterpret_cast<const float4*>(p));
}

// ---- measurement hooks (api.cu) ----
enum Stage {
  kStageKeygen = 0, kStagePass0, kStagePass1, kStagePass2, kStagePass3, kStageCellTables,
  kStageGather, kStageBucketCount, kStageBucketScan, kStageBucketScatter, kStageBucketFinish,
  kStageSlabPartition, kStagePush, kStageSlabExchange, kStageCollide, kNumStages
};
// Multiprocessors of the current device (queried once per device).
int sm_count();
void stage_begin(Stage s, cudaStream_t stream);
void stage_end(Stage s, cudaStream_t stream);
void stage_reset();
void count_launches(int kernels);

// Chained launches.  The kernels of a larger sort call (count, run scan, groups, scatter, finish,
// tail; or the digit passes') run one after the other on one stream, and in the gaps between them
// the next kernel's launch begins when the previous grid has drained.  A kernel launched with
// launch_chained may be set up while its predecessor still runs: every short kernel of the chain
// begins with chain_begin(), which lets the kernel behind it start its launch
// (griddepcontrol.launch_dependents) and then waits until the grids before it are complete
// and their memory visible (griddepcontrol.wait).  Nothing that an earlier kernel of the call writes is
// touched before that wait, so the order of the work is that of the stream.  (The call's inputs, and tables that
// no kernel before writes, may be: a call begins with clear_kernel, an ordinary launch, so that all before
// the call is done; small_sort_kernel and settled_probe_kernel, chained to it, read their particles while
// it runs.)  Launched in the ordinary way
// the same kernels find nothing to wait for.  Kernels that fill the multiprocessors for a long time
// wait with chain_wait() and let the kernel behind them in when a block has done its work
// (chain_release()), or when they end: waiting blocks in their midst cost more than the launch, and blocks that
// are placed while others leave lie unevenly on the multiprocessors, which a kernel whose blocks share
// the work evenly pays for to its end.  Per call, only the short
// kernels chained / these too: without payload 4 M particles 110.8 / 104.0 us, 16 M 348 / 343; with
// payload 1 M 61 / 56, 16 M 556 / 557, 64 M 2241 / 2373, 256 M 10.7 / 11.0 ms.  Without
// payload and without a split, 200 M 6470 / 6810 us.  So they are chained in calls without payload whose
// records are split tile by tile, and in those whose slots are reserved tile by tile.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_begin() {
  chain_release();
  chain_wait();
}

int chained_launches();            // process-wide: 0 none, 1 the short kernels, 2 all
void set_chained_launches(int mode);

template <class... Params, class... Args>
cudaError_t launch_chained_if(bool chained, void (*kernel)(Params...), dim3 grid, dim3 block,
                              size_t shared_bytes, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  cudaLaunchAttribute attribute{};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}
// HEAVY: a kernel that fills the multiprocessors for a long time; chained only in mode 2.
template <bool HEAVY = false, class... Params, class... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes,
                           cudaStream_t stream, Args&&... args) {
  return launch_chained_if(chained_launches() >= (HEAVY ? 2 : 1), kernel, grid, block, shared_bytes,
                           stream, static_cast<Args&&>(args)...);
}

// ---- host-side launchers of the kernels (one translation unit each) ----

// Optional move stage fused into the sort: the sort sees every particle at
// c + v*dt with specular reflection at lo/hi, and the sorted payload carries
// the moved positions and the reflected velocities; the inputs stay as they are.
struct PushSpec {
  int enabled;
  float dt;
  float lo[3], hi[3];
};

// x += v*dt and reflection at the two walls of one axis, in float32 with a rounded
// multiply and a rounded add (fused_particle_push.py:36-44, reference_push :95-108).
// Both wall tests look at the moved coordinate before any reflection.
__device__ __forceinline__ void push_axis(float& c, float& v, float dt, float lo, float hi) {
  c = __fadd_rn(c, __fmul_rn(v, dt));
  const bool below = c < lo, above = c > hi;
  if (below) c = __fsub_rn(__fmul_rn(2.0f, lo), c);
  if (above) c = __fsub_rn(__fmul_rn(2.0f, hi), c);
  if (below || above) v = -v;
}

struct SortArgs {
  const float *x, *y, *z, *velocity;
  int64_t padded, n;
  AetherGrid grid;
  uint64_t seed;
  uint32_t* keys_out;
  int32_t* index_out;
  int32_t *cell_counts, *cell_start;
  float *xs, *ys, *zs, *vs;
  int64_t padded_sorted;
  int64_t num_cells;
  int key_bits;
  void* workspace;
  size_t workspace_bytes;
  cudaStream_t stream;
  PushSpec push;
  int most_blocks;  // 0, or a limit on the blocks of the kernels that work in phases (probe)
  bool zero_padding;  // columns n and on of the sorted velocities become zero
};

size_t standard_workspace_bytes(int64_t n, int64_t num_cells);
size_t standard_workspace_bytes_with_records(int64_t n, int64_t num_cells);
// The digit-pass sort, one launch per step.
cudaError_t standard_sort(const SortArgs& a);
// Arguments of the same sort inside one launch (the hand-over from the bucketed path); refuses the workspaces that standard_sort refuses.
struct DigitPassArgs;
cudaError_t digit_pass_args(const SortArgs& a, DigitPassArgs* out);

// One digit pass over three tiles of zero keys with the ticket dispenser started at 1: the
// tile that would publish first is never processed, so every look-back runs out of polls,
// records kErrLookbackTimeout in the workspace header and returns.  For tests of the give-up
// path; `workspace` needs lookback_probe_workspace_bytes() bytes.
cudaError_t lookback_give_up_probe(void* workspace, size_t workspace_bytes, uint32_t poll_limit,
                                   cudaStream_t stream);
// `blocks` blocks of which each waits, at most `limit_ns`, for one block more; each that gives up
// adds one to *returned.  For tests of the give-up path of the waits between phases, and, with
// `shared_bytes` of shared memory per block, of what runs beside a kernel that stays a while.
constexpr int kProbeMostShared = 200 * 1024;
cudaError_t wait_give_up_probe(void* workspace, size_t workspace_bytes, int blocks,
                               size_t shared_bytes, uint64_t limit_ns, int32_t* returned,
                               cudaStream_t stream);
int64_t lookback_probe_particles();
size_t lookback_probe_workspace_bytes();

struct BucketPlan {
  int shift;          // a bucket is 2^shift consecutive cell ids
  int64_t buckets;
  bool usable;        // false when even single-cell buckets would be too full on average
  bool small_blocks;  // finish kernel shape: two small blocks per multiprocessor, or one large
  bool one_launch;    // small call: one launch
  bool tiled;         // scatter: slots reserved tile by tile
  bool keys_only;     // no payload: 8-byte records and a shape of their own
};
BucketPlan plan_buckets(int64_t n, int64_t num_cells, bool keys_only);
// Most buckets for which the small finish shape is planned (at most 32,768; 0: never).
void set_small_shape_buckets(int64_t buckets);
// Most records of a group of buckets (what one block of the finish kernel sorts at a time).
uint32_t bucket_group_capacity(int64_t n, const BucketPlan& p);
size_t bucketed_workspace_bytes(int64_t n, int64_t num_cells, bool keys_only);
cudaError_t bucketed_sort(const SortArgs& a, const BucketPlan& p);
// Zeroes the padding columns of the sorted velocities in a launch of its own, ahead of all that the call does.
cudaError_t zero_padding_first(const SortArgs& a);

// The bucketed sort of a segmented input, slice by slice (the local sort of the sliced
// multi-GPU exchange): a.n is the CAPACITY of the input arrays, the particle count and the
// segments are read on the device; the bucket plan is made for plan_n particles.
// begin: clears the tables.  slice k: counts, scans and scatters the particles of slice k
// (every source's segment) into chunk k.  finish: bucket starts, groups, and the finish
// kernels; uses a.keys_out ... a.vs.
size_t sliced_sort_workspace_bytes(int64_t capacity, int64_t plan_n, int64_t num_cells, int slices);
cudaError_t sliced_sort_begin(const SortArgs& a, int64_t plan_n, int slices);
cudaError_t sliced_sort_slice(const SortArgs& a, int64_t plan_n, const SliceSegments* segments,
                              int slices, int slice);
cudaError_t sliced_sort_finish(const SortArgs& a, int64_t plan_n, const SliceSegments* segments,
                               int slices);

size_t slab_partition_workspace_bytes(int64_t n, int world);
cudaError_t slab_partition(const float* x, const float* y, const float* z, const float* v,
                           int64_t padded, int64_t n, const AetherGrid& g, int world, float* ox,
                           float* oy, float* oz, float* ovx, float* ovy, float* ovz,
                           int64_t* totals, void* workspace, size_t workspace_bytes,
                           cudaStream_t stream);
cudaError_t launch_make_keys(const float* x, const float* y, const float* z, int64_t n,
                             const AetherGrid& g, uint64_t seed, uint32_t* keys,
                             cudaStream_t stream);
cudaError_t launch_gather(const int32_t* index, int64_t n, const float* x, const float* y,
                          const float* z, const float* velocity, int64_t padded, float* xs,
                          float* ys, float* zs, float* vs, int64_t padded_sorted,
                          cudaStream_t stream);
cudaError_t launch_cell_tables(const uint32_t* sorted_keys, int64_t n, int64_t num_cells,
                               int32_t* cell_counts, int32_t* cell_start, cudaStream_t stream);

cudaError_t slab_exchange_count(const float* x, const float* vx, const PushSpec& push, int64_t n,
                                const AetherGrid& g, int world, int64_t* totals, void* workspace,
                                size_t workspace_bytes, cudaStream_t stream);
// Sliced exchange: one call stores the tiles of one slice and then tells every destination.
struct SliceSignal {
  int slices;
  int slice;
  uint32_t epoch;
  uint32_t* const* peer_flags;    // [world] host array: rank d's flag array [world * slices]
};
cudaError_t slab_exchange_scatter(const float* x, const float* y, const float* z, const float* v,
                                  int64_t padded, int64_t n, const AetherGrid& g, int world,
                                  int rank, float* const* peer_buffers, int64_t capacity,
                                  const int64_t* count_matrix, int32_t* error,
                                  const PushSpec& push, void* workspace, size_t workspace_bytes,
                                  cudaStream_t stream, const SliceSignal* signal = nullptr);
// From the gathered counts matrix[s][k][d] (particles of source s, slice k, for destination d):
// this rank's segment table and the totals totals2d[s][d] the exchange kernel reads.
cudaError_t slab_exchange_prepare(const int64_t* matrix, int world, int slices, int rank,
                                  int64_t* totals2d, SliceSegments* segments, cudaStream_t stream);
void slab_exchange_set_blocks_per_sm(int blocks);
cudaError_t slab_exchange_slice_counts(int64_t n, int world, int slices, int64_t* slice_counts,
                                       void* workspace, size_t workspace_bytes,
                                       cudaStream_t stream);
cudaError_t slab_signal_slice(int world, int rank, int slices, int slice, uint32_t epoch,
                              uint32_t* const* peer_flags, cudaStream_t stream);
cudaError_t slab_wait_slice(const uint32_t* flags, int world, int slices, int slice, uint32_t epoch,
                            uint32_t poll_limit, int32_t* error, cudaStream_t stream);
cudaError_t particle_push(float* x, float* y, float* z, float* vx, float* vy, float* vz, int64_t n,
                          float dt, const float* lo, const float* hi, cudaStream_t stream);
cudaError_t collide_cells(float* velocity, const int* cell_start, float* sigma_g_max,
                          int* collisions, int num_particles, int padded, int num_cells,
                          float selection_factor, float coefficient, float exponent,
                          uint64_t seed, uint64_t step, cudaStream_t stream);

}  // namespace aether
