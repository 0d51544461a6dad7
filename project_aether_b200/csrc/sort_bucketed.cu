// Bucketed path of the particle sort: every byte of particle payload moves
// through HBM twice, both times in full 32-byte sectors or long runs.
//
//   bucket_count_kernel    reads x,y,z once and counts particles per bucket, a
//                          bucket being 2^s consecutive cell ids (the upsweep;
//                          replaces the histogram half of _bin_keys_kernel,
//                          fused_radix_sort.py:106-113)
//   run_scan_kernel        where every (chunk, bucket) run of records starts: the
//                          scatter's write cursors and the finish kernel's table
//   group_kernel           bucket starts, groups of buckets that one block
//                          finishes, where their records lie; decides whether
//                          every bucket can be finished
//   bucket_scatter_kernel  reads x,y,z,v once, builds the key (cell id + Philox
//                          shuffle bits, fused_radix_sort.py:93-103) and writes
//                          one 32-byte record {key, index, x, y, z, vx, vy, vz}
//                          into the particle's bucket
//   tile_scatter_kernel    the same for middling calls, with few buckets: slots
//                          are reserved tile by tile
//   key_split_kernel       calls without payload: 8-byte records {key, index},
//                          put in bucket order tile by tile in shared memory
//   bucket_finish_kernel   a thread block takes a GROUP of consecutive buckets
//                          that fits its shared memory (cut on the device from
//                          the bucket totals, so dense and thin regions both
//                          fill a block): a counting sort on the low key bits
//                          in shared memory, ties put in index order, then
//                          coalesced SoA output of keys, indices, positions,
//                          velocities and the group's rows of cell_counts /
//                          cell_start (replaces the digit passes, the last-pass
//                          count atomics, torch.cumsum and the payload gather:
//                          fused_radix_sort.py:116-203,277-279,
//                          dsmc_gpu_pipeline.py:107-109)
//   bucket_tail_kernel     buckets too large for a group, and the whole digit-pass
//                          sort for calls the bucketed path cannot hold
//   small_sort_kernel      all of the above in one launch, for small calls
//
// The result equals the stable sort by key: the records of a bucket arrive in
// no particular order, and the finish kernel orders them by (low key bits,
// original index), which is the order a stable sort produces.
//
// Record layout of bucket_scatter_kernel: chunk-major (the other scatter kernels write whole
// runs and use one chunk).  The particles are taken in chunks of 2^22
// consecutive indices; the records of chunk c and bucket b form one run, and the
// runs are laid out [chunk][bucket].  While chunk c is being scattered all
// stores fall into its 128 MB region instead of the whole record array: B200
// serves scattered 32-byte stores about 1.6 times faster that way (measured).
// Consecutive buckets are neighbours inside a chunk's region, so a group of
// buckets is still one contiguous run per chunk: the finish kernel collects a
// group with one bulk copy per chunk.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "digit_passes.cuh"

namespace aether {

namespace {

constexpr int kRecordWords = 8;     // 32-byte record {key, index, x, y, z, vx, vy, vz}
constexpr int kKeyRecordWords = 2;  // 8-byte record {key, index} of calls without payload

// Zeroes the header and the counts at the start of a call.  A kernel and not a memset, so that the
// one behind it can be chained to it and is set up, and has loaded its particles, by the time this is
// done.  Per call, memset / this: sort of 5000 particles 19.7 / 18.0 us, gather of 500,000 37.6 / 34.9, of
// 1 M 54.3 / 52.3, step of 200,003 38.5 / 36.0.
// PADDED: also zeroes `columns` columns of three rows `row` apart, from `padding` on (as a launch of its own that cost a
// step of 200,003 particles 2.6 us).  Apart, so that the usual kernel holds few registers: with them the count kernel chained
// to it lay unevenly on the multiprocessors, and a sort of 4 M or 16 M particles took 1 to 2 us more.
template <bool PADDED>
__global__ void __launch_bounds__(512) clear_kernel(uint4* words, int64_t n, float* padding, int64_t row, int64_t columns) {
  chain_release();
  for (int64_t i = blockIdx.x * 512ll + threadIdx.x; i < n; i += gridDim.x * 512ll) words[i] = make_uint4(0u, 0u, 0u, 0u);
  if (PADDED)
    for (int64_t i = blockIdx.x * 512ll + threadIdx.x; i < columns; i += gridDim.x * 512ll)
      padding[i] = padding[row + i] = padding[2 * row + i] = 0.f;
}

// The kernels of a general call that is enqueued behind an attempt to sort a settled state
// (`behind`, see settled_sort.cuh) have nothing to do if that succeeded.  The word they look at is
// final before the first of them runs.
__device__ __forceinline__ bool settled_before(const Header* hdr, bool behind) {
  return behind && ld_relaxed(&hdr->settle_failed) == 0;
}

// ------------------------------------------------------------------------
// Upsweep: particles per bucket.
// ------------------------------------------------------------------------
constexpr int kCountThreads = 512;       // blocks that share an SM (table up to 96 KB)
constexpr int kCountThreadsWide = 1024;  // one block per SM (table up to 200 KB)
constexpr int kCountRounds = 1;          // fewest rounds of four particles per thread for a block

#ifndef AETHER_TUNE_CHUNK_LOG
#define AETHER_TUNE_CHUNK_LOG 22
#endif
constexpr int kChunkLog = AETHER_TUNE_CHUNK_LOG;  // particles per chunk of the record layout at 64 M
                                                  // particles; see chunk_log_for

// Where a block keeps its counts while it works through its particles.
enum CountTable {
  kTableGlobal = 0,    // no table: adds go straight to the chunk's row of counts
  kTableShared32 = 1,  // 32-bit counters in shared memory (up to 200 KB: 51,200 buckets)
  kTableShared16 = 2,  // 16-bit counters, two per word (up to 102,400 buckets)
};
// A 16-bit counter that reaches 2^15 is emptied into the row of counts by the lane whose add took
// it there.  Until that lane has subtracted, the others may add at most what a block counts
// between two barriers (kRoundsPerBarrier rounds of 4096 particles, 2^14), so no counter carries
// into its neighbour however many particles the block counts.
constexpr uint32_t kEmptyAt = 1u << 15;
constexpr int kRoundsPerBarrier = 4;
static_assert(kCountThreadsWide * 4 * kRoundsPerBarrier <= (1 << 15) - 32, "16-bit counters");

template <int TABLE>
__device__ __forceinline__ void table_add(uint32_t* table, uint32_t* row, uint32_t bin, uint32_t count) {
  if (TABLE == kTableShared16) {
    const int sh = 16 * (bin & 1);
    const uint32_t before = (atomicAdd(&table[bin >> 1], count << sh) >> sh) & 0xffffu;
    if (before < kEmptyAt && before + count >= kEmptyAt) {
      atomicSub(&table[bin >> 1], kEmptyAt << sh);
      atomicAdd(&row[bin], kEmptyAt);
    }
  } else {
    atomicAdd(&table[bin], count);
  }
}

// One count per lane into `table`; lanes that hit the same bin share one add when the whole
// warp agrees or (through match.any) when neighbouring lanes do.
// Returns whether lanes shared an add (the same for all lanes): on input in random order
// they never do, and the caller then skips the votes for the rest of its round.
template <int TABLE>
__device__ __forceinline__ bool count_add(uint32_t* table, uint32_t* row, uint32_t bin, bool valid) {
  const uint32_t active = __ballot_sync(0xffffffffu, valid);
  if (active == 0) return true;
  const int first = __ffs(active) - 1;
  const uint32_t first_bin = __shfl_sync(0xffffffffu, bin, first);
  const bool uniform = __all_sync(0xffffffffu, !valid || bin == first_bin);
  if (uniform) {
    if (static_cast<int>(lane_id()) == first) table_add<TABLE>(table, row, first_bin, __popc(active));
    return true;
  }
  const uint32_t next_bin = __shfl_down_sync(0xffffffffu, bin, 1);
  const bool clustered = __any_sync(0xffffffffu, valid && lane_id() < 31 && next_bin == bin);
  if (clustered) {
    const uint32_t peers = __match_any_sync(0xffffffffu, valid ? bin : 0xffffffffu) & active;
    if (valid && (peers & lanemask_lt()) == 0) table_add<TABLE>(table, row, bin, __popc(peers));
  } else if (valid) {
    table_add<TABLE>(table, row, bin, 1u);
  }
  return clustered;
}

// A block counts `per_block` consecutive particles into its table, and adds the table to the
// chunk's row of counts, count[chunk * buckets + b], at the end and wherever its particles pass
// into the next chunk.  One share per block keeps those adds few: with two slices of a chunk per
// block they were more than half as many as the particles at 16 M (16,384 buckets) and more than
// the particles at 256 M (65,536 buckets, whose 16-bit counters also kept the slices below 2^16).
template <int TABLE, bool VEC, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kCountThreads ? 3 : 1)
bucket_count_kernel(const float* __restrict__ x, const float* __restrict__ y,
                    const float* __restrict__ z, const float* __restrict__ v, int64_t padded,
                    PushSpec push, int64_t n, AetherGrid g, int shift, int buckets, int chunk_log,
                    int64_t per_block, uint32_t* __restrict__ bucket_count, Header* hdr,
                    bool behind) {
  chain_begin();
  if (settled_before(hdr, behind)) return;
  extern __shared__ uint32_t hist[];
  const int table_words = TABLE == kTableGlobal ? 0
                          : TABLE == kTableShared16 ? (buckets + 1) / 2 : buckets;
  for (int i = threadIdx.x; i < table_words; i += THREADS) hist[i] = 0;
  __syncthreads();
  // Particle numbers fit 30 bits: index arithmetic in 32.
  int first = static_cast<int>(blockIdx.x * per_block);
  const int block_last = static_cast<int>(min(static_cast<long long>(n), static_cast<long long>(first) + per_block));
  uint32_t shared_rounds = 0;
  while (first < block_last) {
    const int chunk = first >> chunk_log;
    const int last = static_cast<int>(min(static_cast<long long>(block_last),
                                          static_cast<long long>(chunk + 1) << chunk_log));
    uint32_t* row = bucket_count + static_cast<size_t>(chunk) * buckets;
    uint32_t* target = TABLE != kTableGlobal ? hist : row;
    const int rounds = (last - first + THREADS * 4 - 1) / (THREADS * 4);
    for (int r = 0; r < rounds; ++r) {
      const bool whole = VEC && last - first - r * THREADS * 4 >= THREADS * 4;  // no particle missing
      const int i0 = first + (r * THREADS + static_cast<int>(threadIdx.x)) * 4;
      float px[4], py[4], pz[4];
      if (whole) {
        const float4 a = ldcs4(x + i0), b = ldcs4(y + i0), c = ldcs4(z + i0);
        px[0] = a.x; px[1] = a.y; px[2] = a.z; px[3] = a.w;
        py[0] = b.x; py[1] = b.y; py[2] = b.z; py[3] = b.w;
        pz[0] = c.x; pz[1] = c.y; pz[2] = c.z; pz[3] = c.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const bool ok = i0 + k < last;
          px[k] = ok ? x[i0 + k] : 0.f;
          py[k] = ok ? y[i0 + k] : 0.f;
          pz[k] = ok ? z[i0 + k] : 0.f;
        }
      }
      if (push.enabled) {  // count the particles where the fused move stage puts them
        float w[3][4];
        if (whole) {
          const float4 a = ldcs4(v + i0), b = ldcs4(v + padded + i0), c = ldcs4(v + 2 * padded + i0);
          w[0][0] = a.x; w[0][1] = a.y; w[0][2] = a.z; w[0][3] = a.w;
          w[1][0] = b.x; w[1][1] = b.y; w[1][2] = b.z; w[1][3] = b.w;
          w[2][0] = c.x; w[2][1] = c.y; w[2][2] = c.z; w[2][3] = c.w;
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool ok = i0 + k < last;
            w[0][k] = ok ? v[i0 + k] : 0.f;
            w[1][k] = ok ? v[padded + i0 + k] : 0.f;
            w[2][k] = ok ? v[2 * padded + i0 + k] : 0.f;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          push_axis(px[k], w[0][k], push.dt, push.lo[0], push.hi[0]);
          push_axis(py[k], w[1][k], push.dt, push.lo[1], push.hi[1]);
          push_axis(pz[k], w[2][k], push.dt, push.lo[2], push.hi[2]);
        }
      }
      bool sharing = true;  // the round's first particle tells whether votes are worth it
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t bin = cell_of(px[k], py[k], pz[k], g) >> shift;
        const bool valid = whole || i0 + k < last;
        if (sharing) sharing = count_add<TABLE>(target, row, bin, valid);
        else if (valid) table_add<TABLE>(target, row, bin, 1u);
      }
      shared_rounds += sharing;
      if (TABLE == kTableShared16 && (r + 1) % kRoundsPerBarrier == 0) __syncthreads();
    }
    if (TABLE != kTableGlobal) {
      __syncthreads();
      for (int i = threadIdx.x; i < table_words; i += THREADS) {
        const uint32_t w = hist[i];
        if (w) {
          if (TABLE == kTableShared16) {
            if (w & 0xffffu) atomicAdd(&row[2 * i], w & 0xffffu);
            if (w >> 16) atomicAdd(&row[2 * i + 1], w >> 16);
          } else {
            atomicAdd(&row[i], w);
          }
          hist[i] = 0;
        }
      }
      __syncthreads();
    }
    first = last;
  }
  // What the block's first warp has seen tells the scatter whether the input is in some order.
  if (threadIdx.x == 0 && shared_rounds) atomicAdd(&hdr->shared_rounds, shared_rounds);
}

// ------------------------------------------------------------------------
// Where the runs start.
// ------------------------------------------------------------------------
constexpr int kRunScanThreads = 1024;
constexpr int kRunScanPart = kRunScanThreads * 4;  // entries of a row per block

// Exclusive scan of every chunk's row of counts; block (part, chunk) writes kRunScanPart entries
// of the row.  Chunk c's records begin at record c << chunk_log, because a chunk is that many
// consecutive particles, so the rows do not wait for one another; and a block adds up the
// entries before its own for itself (they lie in L2) instead of waiting for their blocks.  The
// starts are written twice: as the scatter's cursors, which the scatter advances, and as the
// table run_begin[chunk * buckets + b] (with n behind its last entry) from which the run of any
// range of buckets [b0, b1) in chunk c is taken: run_begin[c*B + b0] .. run_begin[c*B + b1].
// Bound by latency.  This kernel and group_kernel replace seven (bucket totals, two bucket scans,
// three levels of run scan, two group kernels); from the count's end to the scatter's begin, before
// and after: 4 M particles in 10,000 cells 75 / 10 us, 16 M in 2 M 33 / 15, 128 M in 16 M 89 / 36.
__global__ void __launch_bounds__(kRunScanThreads)
run_scan_kernel(const uint32_t* __restrict__ count, int buckets, int chunk_log, uint32_t n,
                uint32_t* __restrict__ cursor, uint32_t* __restrict__ run_begin, const Header* hdr,
                bool behind) {
  chain_begin();
  if (settled_before(hdr, behind)) return;
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t total, before_part;
  const int tid = threadIdx.x, lane = tid & 31;
  const size_t row = static_cast<size_t>(blockIdx.y) * buckets;
  const int part = blockIdx.x * kRunScanPart;
  const int i = part + tid * 4;
  const bool vec = buckets % 4 == 0;  // rows then start on 16-byte boundaries
  if (tid == 0) before_part = static_cast<uint32_t>(blockIdx.y) << chunk_log;
  uint32_t c[4] = {0, 0, 0, 0}, before = 0;
  if (vec) {
    if (i < buckets) {
      const uint4 q = *reinterpret_cast<const uint4*>(count + row + i);
      c[0] = q.x; c[1] = q.y; c[2] = q.z; c[3] = q.w;
    }
#pragma unroll 8
    for (int k = tid * 4; k < part; k += kRunScanPart) {
      const uint4 q = *reinterpret_cast<const uint4*>(count + row + k);
      before += q.x + q.y + q.z + q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = i + k < buckets ? count[row + i + k] : 0u;
#pragma unroll 8
    for (int k = tid; k < part; k += kRunScanThreads) before += count[row + k];
  }
  before = __reduce_add_sync(0xffffffffu, before);
  __syncthreads();
  if (lane == 0 && before) atomicAdd(&before_part, before);
  uint32_t start = block_exclusive_scan(c[0] + c[1] + c[2] + c[3], warp_sum, &total);
  start += before_part;  // complete: the scan has barriers
  if (vec) {
    if (i < buckets) {
      const uint4 q = make_uint4(start, start + c[0], start + c[0] + c[1], start + c[0] + c[1] + c[2]);
      *reinterpret_cast<uint4*>(cursor + row + i) = q;
      *reinterpret_cast<uint4*>(run_begin + row + i) = q;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < buckets) {
        cursor[row + i + k] = start;
        run_begin[row + i + k] = start;
      }
      start += c[k];
    }
  }
  if (blockIdx.x == 0 && blockIdx.y == gridDim.y - 1 && tid == 0)
    run_begin[static_cast<size_t>(gridDim.y) * buckets] = n;
}

// ------------------------------------------------------------------------
// Scatter of 32-byte records into buckets.
// ------------------------------------------------------------------------
constexpr int kScatterThreads = 512;

__device__ __forceinline__ void store_record(uint32_t* dst, uint32_t key, uint32_t index, float x,
                                             float y, float z, float vx, float vy, float vz) {
  // One full 32-byte sector per record.
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(key),
               "r"(index), "r"(__float_as_uint(x)), "r"(__float_as_uint(y)),
               "r"(__float_as_uint(z)), "r"(__float_as_uint(vx)), "r"(__float_as_uint(vy)),
               "r"(__float_as_uint(vz))
               : "memory");
}

// Reserves one slot in bucket `b`.  Lanes that target the same bucket share one
// atomic: always when the whole warp agrees (cell-sorted input), and through
// match.any when at least two neighbouring lanes agree (nearly sorted input).
// Random input, where no neighbours agree, goes straight to one atomic per lane.
__device__ __forceinline__ uint32_t reserve_slot(uint32_t* cursor, uint32_t b, bool valid) {
  const uint32_t active = __ballot_sync(0xffffffffu, valid);
  if (active == 0) return 0;
  const int first = __ffs(active) - 1;
  const uint32_t first_b = __shfl_sync(0xffffffffu, b, first);
  const bool uniform = __all_sync(0xffffffffu, !valid || b == first_b);
  uint32_t slot = 0;
  if (uniform) {
    if (static_cast<int>(lane_id()) == first) slot = atomicAdd(&cursor[first_b], __popc(active));
    return __shfl_sync(0xffffffffu, slot, first) + __popc(active & lanemask_lt());
  }
  const uint32_t next_b = __shfl_down_sync(0xffffffffu, b, 1);
  const bool clustered = __any_sync(0xffffffffu, valid && lane_id() < 31 && next_b == b);
  if (clustered) {
    const uint32_t peers = __match_any_sync(0xffffffffu, valid ? b : 0xffffffffu) & active;
    const int leader = __ffs(peers) - 1;
    if (valid && static_cast<int>(lane_id()) == leader) slot = atomicAdd(&cursor[b], __popc(peers));
    slot = __shfl_sync(0xffffffffu, slot, leader < 0 ? 0 : leader) + __popc(peers & lanemask_lt());
    return slot;
  }
  if (valid) slot = atomicAdd(&cursor[b], 1u);
  return slot;
}

// ITEMS consecutive particles per thread and round (4: 128-bit loads, 2: 64-bit
// loads with twice the resident threads to keep more slot reservations in flight).
template <int ITEMS>
__device__ __forceinline__ void load_items(const float* p, float* out) {
  static_assert(ITEMS == 4 || ITEMS == 2, "one access");
  if (ITEMS == 4) {
    const float4 a = ldcs4(p);
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
  } else {
    const float2 a = __ldcs(reinterpret_cast<const float2*>(p));
    out[0] = a.x; out[1] = a.y;
  }
}

// Input in some order (the count kernel's first warps have seen neighbours in one bucket in `some_order` rounds), input
// in none, or any.
enum ScatterOnly { kScatterAny, kScatterOrdered, kScatterRandom };

template <bool VEC, int ITEMS, int RECORD_WORDS>
__global__ void __launch_bounds__(kScatterThreads, 8 / ITEMS)
bucket_scatter_kernel(const float* __restrict__ x, const float* __restrict__ y,
                      const float* __restrict__ z, const float* __restrict__ v, int64_t padded,
                      PushSpec push, int64_t n, AetherGrid g, uint32_t k0, uint32_t k1, int shift,
                      int buckets, int chunk_log, uint32_t* __restrict__ cursor,
                      uint32_t* __restrict__ records, const Header* __restrict__ hdr,
                      ScatterOnly only, uint32_t some_order, bool behind) {
  chain_wait();
  if (settled_before(hdr, behind) || hdr->use_standard) return;
  if (only != kScatterAny && (hdr->shared_rounds >= some_order) != (only == kScatterOrdered)) return;
  const int64_t groups = (n + ITEMS - 1) / ITEMS;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kScatterThreads;
  const int64_t rounds = (groups + stride - 1) / stride;
  for (int64_t r = 0; r < rounds; ++r) {
    const int64_t i0 = (r * stride + static_cast<int64_t>(blockIdx.x) * kScatterThreads +
                        threadIdx.x) * ITEMS;
    float f[6][ITEMS];
    if (VEC && i0 + ITEMS <= n) {
      load_items<ITEMS>(x + i0, f[0]);
      load_items<ITEMS>(y + i0, f[1]);
      load_items<ITEMS>(z + i0, f[2]);
      if (v) {
        load_items<ITEMS>(v + i0, f[3]);
        load_items<ITEMS>(v + padded + i0, f[4]);
        load_items<ITEMS>(v + 2 * padded + i0, f[5]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        const bool ok = i0 + k < n;
        f[0][k] = ok ? x[i0 + k] : 0.f;
        f[1][k] = ok ? y[i0 + k] : 0.f;
        f[2][k] = ok ? z[i0 + k] : 0.f;
        f[3][k] = ok && v ? v[i0 + k] : 0.f;
        f[4][k] = ok && v ? v[padded + i0 + k] : 0.f;
        f[5][k] = ok && v ? v[2 * padded + i0 + k] : 0.f;
      }
    }
    if (!v) {
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) f[3][k] = f[4][k] = f[5][k] = 0.f;
    }
    if (push.enabled) {  // the fused move stage: the record carries the moved particle
#pragma unroll
      for (int k = 0; k < ITEMS; ++k) {
        push_axis(f[0][k], f[3][k], push.dt, push.lo[0], push.hi[0]);
        push_axis(f[1][k], f[4][k], push.dt, push.lo[1], push.hi[1]);
        push_axis(f[2][k], f[5][k], push.dt, push.lo[2], push.hi[2]);
      }
    }
    uint32_t key[ITEMS], slot[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const uint32_t cell = cell_of(f[0][k], f[1][k], f[2][k], g);
      const uint32_t run = static_cast<uint32_t>((i0 + k) >> chunk_log) * buckets + (cell >> shift);
      slot[k] = reserve_slot(cursor, run, i0 + k < n);
      key[k] = make_key(cell, static_cast<uint32_t>(i0 + k), k0, k1);
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
      if (RECORD_WORDS == kKeyRecordWords) {
        if (i0 + k < n)
          reinterpret_cast<uint2*>(records)[slot[k]] = make_uint2(key[k], static_cast<uint32_t>(i0 + k));
      } else if (i0 + k < n)
        store_record(records + static_cast<size_t>(slot[k]) * kRecordWords, key[k],
                     static_cast<uint32_t>(i0 + k), f[0][k], f[1][k], f[2][k], f[3][k], f[4][k],
                     f[5][k]);
  }
  chain_release();
}

// Lanes of a warp that do not agree on a bucket skip the votes for the rest of a tile.
__device__ __forceinline__ uint32_t rank_in_tile(uint32_t* table, uint32_t b, bool valid, bool& sharing) {
  if (!sharing) return valid ? atomicAdd(&table[b], 1u) : 0u;
  const uint32_t next_b = __shfl_down_sync(0xffffffffu, b, 1);
  sharing = __any_sync(0xffffffffu, valid && lane_id() < 31 && next_b == b);
  return reserve_slot(table, b, valid);
}

// ------------------------------------------------------------------------
// Scatter of middling inputs: slots reserved tile by tile.
// ------------------------------------------------------------------------
// With a thousand buckets or so the slot counters fill few L2 lines, and one returning add per
// particle queues on them (1 M particles on 2048 counters: 47 us).  Here a block ranks a tile's
// particles with adds in shared memory and reserves each bucket's slots with one add per tile,
// consecutive threads on consecutive counters: 17 us, the rate of scattered 32-byte stores
// (62 G/s).  It pays while a tile has about as many particles as there are buckets.  Staging the
// tile in shared memory, so that a bucket's records leave side by side, took 23 us.
// us per call as blocks of 512 threads, two per multiprocessor, that stay and take tiles in turn / one tile each, the next
// block placed as one ends / 1024 threads, one tile each: 650,000 particles 47.0 / 45.1 / 47.1, 1 M 53.7 / 51.3 / 51.4,
// 2 M 95.2 / 90.9 / 90.5, 4 M 158.5 / 157.1 / 153.5, 6 M 216 / 216 / 210; 512 threads with eight
// particles each, one block per multiprocessor (as it was from 1.2 M on) 2 M 97, 4 M 167, 6 M 231.  Behind a sort of a
// settled state, where the kernel usually returns at once, blocks stay.
template <bool VEC, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
tile_scatter_kernel(const float* __restrict__ x, const float* __restrict__ y,
                    const float* __restrict__ z, const float* __restrict__ v, int64_t padded,
                    PushSpec push, int64_t n, AetherGrid g, uint32_t k0, uint32_t k1, int shift,
                    int buckets, int chunk_log, uint32_t* __restrict__ cursor,
                    uint32_t* __restrict__ records, const Header* __restrict__ hdr,
                    bool behind) {
  constexpr int kItems = 4, kTile = THREADS * kItems;
  chain_wait();
  if (settled_before(hdr, behind) || hdr->use_standard) return;
  extern __shared__ uint32_t slot_of[];  // a tile's counts, then its first slots
  const int tid = threadIdx.x;
  const int64_t tiles = (n + kTile - 1) / kTile;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t first = tile * kTile;
    uint32_t* row = cursor + static_cast<size_t>(first >> chunk_log) * buckets;
    for (int b = tid; b < buckets; b += THREADS) slot_of[b] = 0;
    __syncthreads();
    float f[6][kItems];
    uint32_t key[kItems], rank[kItems];
    bool sharing = true;
    const int64_t i0 = first + tid * 4;
    if (VEC && i0 + 4 <= n) {
      load_items<4>(x + i0, f[0]);
      load_items<4>(y + i0, f[1]);
      load_items<4>(z + i0, f[2]);
      if (v) {
        load_items<4>(v + i0, f[3]);
        load_items<4>(v + padded + i0, f[4]);
        load_items<4>(v + 2 * padded + i0, f[5]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = i0 + k < n;
        f[0][k] = ok ? x[i0 + k] : 0.f;
        f[1][k] = ok ? y[i0 + k] : 0.f;
        f[2][k] = ok ? z[i0 + k] : 0.f;
        f[3][k] = ok && v ? v[i0 + k] : 0.f;
        f[4][k] = ok && v ? v[padded + i0 + k] : 0.f;
        f[5][k] = ok && v ? v[2 * padded + i0 + k] : 0.f;
      }
    }
    if (!v) {
#pragma unroll
      for (int k = 0; k < 4; ++k) f[3][k] = f[4][k] = f[5][k] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int64_t i = i0 + k;
      if (push.enabled) {  // the fused move stage: the record carries the moved particle
        push_axis(f[0][k], f[3][k], push.dt, push.lo[0], push.hi[0]);
        push_axis(f[1][k], f[4][k], push.dt, push.lo[1], push.hi[1]);
        push_axis(f[2][k], f[5][k], push.dt, push.lo[2], push.hi[2]);
      }
      const uint32_t cell = cell_of(f[0][k], f[1][k], f[2][k], g);
      key[k] = make_key(cell, static_cast<uint32_t>(i), k0, k1);
      rank[k] = rank_in_tile(slot_of, cell >> shift, i < n, sharing);
    }
    __syncthreads();
#pragma unroll 4
    for (int b = tid; b < buckets; b += THREADS) {
      const uint32_t c = slot_of[b];
      if (c) slot_of[b] = atomicAdd(&row[b], c);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int64_t i = i0 + k;
      if (i < n)
        store_record(records + static_cast<size_t>(slot_of[key[k] >> (kShuffleBits + shift)] + rank[k]) *
                                   kRecordWords,
                     key[k], static_cast<uint32_t>(i), f[0][k], f[1][k], f[2][k], f[3][k], f[4][k],
                     f[5][k]);
    }
    __syncthreads();  // the table is reused by the next tile
  }
  chain_release();
}

// ------------------------------------------------------------------------
// Calls without payload: 8-byte records, split tile by tile.
// ------------------------------------------------------------------------
// A record per particle is a quarter of the payload's, so a finish block holds large buckets
// and a call has few of them: few enough to put a tile of particles in bucket order in shared
// memory and write it out in runs.  Per tile: ranks from returning adds in shared memory, one
// add per bucket and tile on the slot counters in L2 (consecutive threads, consecutive
// counters), places from a scan while those are under way, records staged by place, then
// written out with neighbouring lanes at neighbouring addresses.  The scatter kernel above
// instead pays one returning L2 add and one store request per particle (64 G/s at best).
// Bound by instructions and latency (32 warps per multiprocessor between barriers): 4 M particles
// on 1250 buckets 37 us, 16 M on 4096 155, where the 32-byte records took 93 and 241 (before a tile was
// written out beside the next one's count, see kSplitHeld).
constexpr int kSplitThreads = 512;       // two blocks per multiprocessor
constexpr int kSplitThreadsWide = 1024;  // one block, twice the tile
constexpr int kSplitMaxBuckets = 16384;  // 128 KB of tables beside the stage
// HELD: up to this many buckets per thread what the adds on the slot counters return stays in registers
// until the scan is done, and the next tile's first positions are loaded while a tile is written
// out.  Whole call, without / with: 1 M particles 43.1 / 41.1 us, 4 M 94.8 / 94.0, 8 M 172.0 / 168.0, 16 M 338.7 /
// 333.4.  With more buckets the registers would spill: nothing is held, and a tile is cleared, counted and
// written out one after the other (8192 buckets: 30 M 661 us, 45 M 1218; with the table cleared ahead of the
// write-out there too 666 and 1234).
constexpr int kSplitHeld = 4;

__host__ __device__ inline size_t split_smem_bytes(int tile, int buckets) {
  return static_cast<size_t>(tile) * 8 + 2 * (static_cast<size_t>(buckets + 3) / 4 * 4) * sizeof(uint32_t);
}

template <bool VEC, int ITEMS, int THREADS, bool HELD>
__global__ void __launch_bounds__(THREADS, THREADS <= 512 ? 2 : 1)
key_split_kernel(const float* __restrict__ x, const float* __restrict__ y,
                 const float* __restrict__ z, int64_t n, AetherGrid g, uint32_t k0, uint32_t k1,
                 int shift, int buckets, int chunk_log, int tile, uint32_t* __restrict__ cursor,
                 uint2* __restrict__ records, const Header* __restrict__ hdr) {
  static_assert(ITEMS % 4 == 0, "whole 16-byte loads");
  constexpr int kTile = THREADS * ITEMS;
  chain_wait();
  if (hdr->use_standard) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint32_t warp_sum[2][32];
  uint2* stage = reinterpret_cast<uint2*>(smem_raw);
  uint32_t* place = reinterpret_cast<uint32_t*>(stage + kTile);  // counts, then first places
  const int table = (buckets + 3) / 4 * 4;
  uint32_t* to_slot = place + table;  // slot minus place of a bucket's records
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Particle numbers fit 30 bits: index arithmetic in 32.
  const int last = static_cast<int>(n);
  const int stride = gridDim.x * tile;
  static_assert(kTile <= 1 << 16, "ranks of 16 bits");
  float px[ITEMS], py[ITEMS], pz[ITEMS];
  auto load_four = [&](int first, int q) {
    const int at = (q / 4 * THREADS + tid) * 4, i0 = first + at;
    if (VEC && at < tile && last - first >= tile) {  // the same for a whole warp: tiles are multiples of 128
      load_items<4>(x + i0, px + q);
      load_items<4>(y + i0, py + q);
      load_items<4>(z + i0, pz + q);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = at < tile && i0 + k < last;
        px[q + k] = ok ? x[i0 + k] : 0.f;
        py[q + k] = ok ? y[i0 + k] : 0.f;
        pz[q + k] = ok ? z[i0 + k] : 0.f;
      }
    }
  };
  auto clear_counts = [&] {
    for (int b = tid * 4; b < table; b += THREADS * 4)
      *reinterpret_cast<uint4*>(&place[b]) = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
  };
  int first = blockIdx.x * tile;
  if (HELD && first < last) load_four(first, 0);
  if (HELD) clear_counts();
  for (; first < last; first += stride) {
    if (!HELD) clear_counts();
    uint32_t* row = cursor + static_cast<size_t>(first >> chunk_log) * buckets;
    const int end = min(last, first + tile);
    uint32_t key[ITEMS], ranks[ITEMS / 2];  // two ranks of 16 bits to a word
    bool sharing = true;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      if (!HELD && k % 4 == 0) load_four(first, k);
      const int i = first + (k / 4 * THREADS + tid) * 4 + k % 4;
      const uint32_t cell = cell_of(px[k], py[k], pz[k], g);
      key[k] = make_key(cell, static_cast<uint32_t>(i), k0, k1);
      const uint32_t rank = rank_in_tile(place, cell >> shift, i < end, sharing);
      ranks[k / 2] = k % 2 ? ranks[k / 2] | rank << 16 : rank;
      if (HELD && k % 4 == 3 && k + 1 < ITEMS) load_four(first, k + 1);
    }
    __syncthreads();  // the tile is counted, and the one before it written out
    uint32_t got[kSplitHeld] = {};
    if (HELD) {
#pragma unroll
      for (int k = 0; k < kSplitHeld; ++k) {
        const int b = tid + k * THREADS;
        const uint32_t c = b < buckets ? place[b] : 0u;
        if (c) got[k] = atomicAdd(&row[b], c);
      }
    } else {
#pragma unroll 8
      for (int b = tid; b < buckets; b += THREADS) {
        const uint32_t c = place[b];
        to_slot[b] = c ? atomicAdd(&row[b], c) : 0u;
      }
      __syncthreads();
    }
    // Exclusive scan of the counts, in place: four buckets per thread and step.  (The adds above have
    // read the counts before the first step's barrier.)
    uint32_t carry = 0;
    for (int base = 0, set = 0; base < table; base += THREADS * 4, set ^= 1) {
      const int b = base + tid * 4;
      uint4 c = make_uint4(0u, 0u, 0u, 0u);
      if (b < table) c = *reinterpret_cast<const uint4*>(&place[b]);
      const uint32_t sum = c.x + c.y + c.z + c.w;
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      if (lane == 31) warp_sum[set][warp] = incl;
      __syncthreads();
      uint32_t sums = lane < THREADS / 32 ? warp_sum[set][lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, sums, o);
        if (lane >= o) sums += up;
      }
      const uint32_t before_warp = __shfl_sync(0xffffffffu, sums, (warp + 31) & 31);
      const uint32_t start = carry + (warp ? before_warp : 0u) + incl - sum;
      if (b < table)
        *reinterpret_cast<uint4*>(&place[b]) =
            make_uint4(start, start + c.x, start + c.x + c.y, start + c.x + c.y + c.z);
      carry += __shfl_sync(0xffffffffu, sums, 31);
    }
    __syncthreads();
    if (HELD) {
#pragma unroll
      for (int k = 0; k < kSplitHeld; ++k) {
        const int b = tid + k * THREADS;
        if (b < buckets) to_slot[b] = got[k] - place[b];
      }
    } else {
      for (int b = tid; b < buckets; b += THREADS) to_slot[b] -= place[b];
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const int i = first + (k / 4 * THREADS + tid) * 4 + k % 4;
      if (i < end)
        stage[place[key[k] >> (kShuffleBits + shift)] + (k % 2 ? ranks[k / 2] >> 16 : ranks[k / 2] & 0xffffu)] =
            make_uint2(key[k], static_cast<uint32_t>(i));
    }
    __syncthreads();
    // The next tile's first positions are on their way while this one is written out, and the writes
    // while the next one is counted.
    if (HELD) {
      if (first + stride < last) load_four(first + stride, 0);
      clear_counts();
    }
    const int here = end - first;
#pragma unroll 4
    for (int j = tid; j < here; j += THREADS) {
      const uint2 r = stage[j];
      records[to_slot[r.x >> (kShuffleBits + shift)] + static_cast<uint32_t>(j)] = r;
    }
    if (!HELD) __syncthreads();  // the tables and the stage are reused by the next tile
  }
  chain_release();
}

// ------------------------------------------------------------------------
// Segmented input (the local sort of the sliced multi-GPU exchange): the particles of one
// slice are up to kMaxWorld index ranges of the input arrays, known on the device only.
// ------------------------------------------------------------------------
constexpr int kSegmentUnit = 16384;  // particles per work unit of the segment kernels

// Work unit `unit` of slice `k`: the units of source 0's segment, then source 1's, ...  Each
// segment is cut from its 4-aligned start in pieces of kSegmentUnit, so that the 16-byte loads
// stay aligned.  Returns false past the last unit; else [first, last) is the piece (first a
// multiple of 4) and `lo` the first index in it that belongs to the segment.
__device__ __forceinline__ bool segment_unit(const SliceSegments* __restrict__ seg, int k, int unit,
                                             int64_t* first, int64_t* last, int64_t* lo) {
  const int sources = static_cast<int>(seg->sources);
  for (int s = 0; s < sources; ++s) {
    const int64_t begin = seg->first[k][s], length = seg->length[k][s];
    if (length == 0) continue;
    const int64_t base = begin & ~int64_t{3};
    const int units = static_cast<int>((begin + length - base + kSegmentUnit - 1) / kSegmentUnit);
    if (unit < units) {
      *first = base + static_cast<int64_t>(unit) * kSegmentUnit;
      *last = min(static_cast<long long>(begin + length), static_cast<long long>(*first + kSegmentUnit));
      *lo = max(static_cast<long long>(begin), static_cast<long long>(*first));
      return true;
    }
    unit -= units;
  }
  return false;
}

// Particles per bucket of one slice, added to the slice's row of counts.  `capacity` is the
// length of the input arrays (vector loads must not pass it).
template <int TABLE, int THREADS>
__global__ void __launch_bounds__(THREADS)
bucket_count_segments_kernel(const float* __restrict__ x, const float* __restrict__ y,
                             const float* __restrict__ z, int64_t capacity, bool vec,
                             const SliceSegments* __restrict__ seg, int k, AetherGrid g, int shift,
                             int buckets, uint32_t* __restrict__ row) {
  extern __shared__ uint32_t hist[];
  if (TABLE != kTableGlobal) {
    for (int i = threadIdx.x; i < buckets; i += THREADS) hist[i] = 0;
    __syncthreads();
  }
  uint32_t* target = TABLE != kTableGlobal ? hist : row;
  int64_t first, last, lo;
  for (int unit = blockIdx.x; segment_unit(seg, k, unit, &first, &last, &lo); unit += gridDim.x) {
    // Every thread of the block makes the same number of rounds: the adds below use
    // warp-wide votes, which all 32 lanes must reach.
    for (int64_t round = first; round < last; round += THREADS * 4) {
      const int64_t i0 = round + static_cast<int64_t>(threadIdx.x) * 4;
      float px[4], py[4], pz[4];
      if (vec && i0 + 4 <= capacity) {
        const float4 a = ldcs4(x + i0), b = ldcs4(y + i0), c = ldcs4(z + i0);
        px[0] = a.x; px[1] = a.y; px[2] = a.z; px[3] = a.w;
        py[0] = b.x; py[1] = b.y; py[2] = b.z; py[3] = b.w;
        pz[0] = c.x; pz[1] = c.y; pz[2] = c.z; pz[3] = c.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool ok = i0 + j >= lo && i0 + j < last;
          px[j] = ok ? x[i0 + j] : 0.f;
          py[j] = ok ? y[i0 + j] : 0.f;
          pz[j] = ok ? z[i0 + j] : 0.f;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        count_add<TABLE>(target, row, cell_of(px[j], py[j], pz[j], g) >> shift,
                         i0 + j >= lo && i0 + j < last);
    }
  }
  if (TABLE != kTableGlobal) {
    __syncthreads();
    for (int i = threadIdx.x; i < buckets; i += THREADS)
      if (hist[i]) atomicAdd(&row[i], hist[i]);
  }
}

// Exclusive scan of one slice's row of counts, offset by the records of the slices before it:
// the scatter's cursors and the finish kernel's run_begin row of that chunk.  One block.
// STAGED: the row fits shared memory (padded against bank conflicts); it is read and written
// once, coalesced, and every thread scans a contiguous piece of it.  Otherwise 1024 entries
// at a time.
constexpr int kFlatScanBlock = 1024;
constexpr int kStagedScanMax = 48 * 1024;  // buckets whose row (plus padding) fits 200 KB

template <bool STAGED>
__global__ void __launch_bounds__(kFlatScanBlock)
chunk_scan_kernel(const uint32_t* __restrict__ row, int buckets,
                  const SliceSegments* __restrict__ seg, int k, uint32_t* __restrict__ cursor_row,
                  uint32_t* __restrict__ run_begin_row) {
  extern __shared__ uint32_t staged[];
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t total, carry;
  if (STAGED) {
    const int per = (buckets + kFlatScanBlock - 1) / kFlatScanBlock;
    const int pad = 1 + (per & 1);  // pieces an odd number of words apart: no bank conflicts
    auto at = [per, pad](int i) { return i + i / per * pad; };
    for (int i = threadIdx.x; i < buckets; i += kFlatScanBlock) staged[at(i)] = row[i];
    __syncthreads();
    const int first = min(buckets, static_cast<int>(threadIdx.x) * per);
    const int last = min(buckets, first + per);
    uint32_t sum = 0;
    for (int b = first; b < last; ++b) sum += staged[at(b)];
    uint32_t run = seg->chunk_base[k] + block_exclusive_scan(sum, warp_sum, &total);
    for (int b = first; b < last; ++b) {
      const uint32_t here = staged[at(b)];
      staged[at(b)] = run;
      run += here;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < buckets; i += kFlatScanBlock) {
      const uint32_t start = staged[at(i)];
      cursor_row[i] = start;
      run_begin_row[i] = start;
    }
  } else {
    if (threadIdx.x == 0) carry = seg->chunk_base[k];
    __syncthreads();
    for (int base = 0; base < buckets; base += kFlatScanBlock) {
      const int i = base + threadIdx.x;
      const uint32_t v = i < buckets ? row[i] : 0u;
      const uint32_t excl = block_exclusive_scan(v, warp_sum, &total);
      if (i < buckets) {
        cursor_row[i] = carry + excl;
        run_begin_row[i] = carry + excl;
      }
      __syncthreads();
      if (threadIdx.x == 0) carry += total;
      __syncthreads();
    }
  }
  // Behind the last chunk's row: the end of the last run.
  if (k + 1 == static_cast<int>(seg->slices) && threadIdx.x == 0) run_begin_row[buckets] = seg->n;
}

// Records of one slice into the runs of chunk k.
template <int ITEMS>
__global__ void __launch_bounds__(kScatterThreads, 8 / ITEMS)
bucket_scatter_segments_kernel(const float* __restrict__ x, const float* __restrict__ y,
                               const float* __restrict__ z, const float* __restrict__ v,
                               int64_t padded, int64_t capacity, bool vec,
                               const SliceSegments* __restrict__ seg, int k, AetherGrid g,
                               uint32_t k0, uint32_t k1, int shift, int buckets,
                               uint32_t* __restrict__ cursor_row, uint32_t* __restrict__ records) {
  int64_t first, last, lo;
  for (int unit = blockIdx.x; segment_unit(seg, k, unit, &first, &last, &lo); unit += gridDim.x) {
    // Every thread of the block makes the same number of rounds: the slot reservation uses
    // warp-wide votes, which all 32 lanes must reach.
    for (int64_t round = first; round < last; round += kScatterThreads * ITEMS) {
      const int64_t i0 = round + static_cast<int64_t>(threadIdx.x) * ITEMS;
      float f[6][ITEMS];
      if (vec && i0 + ITEMS <= capacity) {
        load_items<ITEMS>(x + i0, f[0]);
        load_items<ITEMS>(y + i0, f[1]);
        load_items<ITEMS>(z + i0, f[2]);
        load_items<ITEMS>(v + i0, f[3]);
        load_items<ITEMS>(v + padded + i0, f[4]);
        load_items<ITEMS>(v + 2 * padded + i0, f[5]);
      } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
          const bool ok = i0 + j >= lo && i0 + j < last;
          f[0][j] = ok ? x[i0 + j] : 0.f;
          f[1][j] = ok ? y[i0 + j] : 0.f;
          f[2][j] = ok ? z[i0 + j] : 0.f;
          f[3][j] = ok ? v[i0 + j] : 0.f;
          f[4][j] = ok ? v[padded + i0 + j] : 0.f;
          f[5][j] = ok ? v[2 * padded + i0 + j] : 0.f;
        }
      }
      uint32_t key[ITEMS], slot[ITEMS];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const bool ok = i0 + j >= lo && i0 + j < last;
        const uint32_t cell = cell_of(f[0][j], f[1][j], f[2][j], g);
        slot[j] = reserve_slot(cursor_row, cell >> shift, ok);
        key[j] = make_key(cell, static_cast<uint32_t>(i0 + j), k0, k1);
      }
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (i0 + j >= lo && i0 + j < last)
          store_record(records + static_cast<size_t>(slot[j]) * kRecordWords, key[j],
                       static_cast<uint32_t>(i0 + j), f[0][j], f[1][j], f[2][j], f[3][j], f[4][j],
                       f[5][j]);
    }
  }
}

// ------------------------------------------------------------------------
// Groups: consecutive buckets that one block finishes together.
// ------------------------------------------------------------------------
// Words of one row of a group's table: one entry per chunk and three more, rounded up to
// whole 16-byte pieces (the finish kernel fetches the tables with 16-byte copies).
__host__ __device__ inline int table_row_words(int chunks) { return (chunks + 3 + 3) / 4 * 4; }

constexpr int kGroupSpanLog = 8;
constexpr int kGroupSpan = 1 << kGroupSpanLog;  // buckets per block of group_kernel
// Up to here a block of group_kernel adds up the counts before its own, 32 loads per thread at most (measured
// up to some 5500 buckets, 5 M particles with payload: 201.0 us with the run scan, 199.8 without).
constexpr int kMostOneChunkBuckets = 8192;
constexpr int kGroupStagedChunks = 32;  // chunks whose run starts the block keeps

// What a block of group_kernel keeps while it cuts its buckets into groups.
struct GroupCut {
  uint32_t start[kGroupSpan + 1];  // records before each of the block's buckets
  uint16_t link[kGroupSpan];       // where a group that began with this bucket would end
  uint16_t group_first[kGroupSpan], jumps[kGroupSpan + 1];
  unsigned char is_first[kGroupSpan + 1];
  uint32_t warp_sum[32], found, list_base, found_other, other_base;
};

// Cuts every block of the `here` buckets (from one that is `first_of_block` to its `block_end`, `longest` buckets at most) greedily
// into groups of at most `most` consecutive buckets with at most `capacity` records (each bucket looks up where a group
// that began with it would end, and those links are followed).  Afterwards group k of the block,
// k < c.found, has the buckets c.group_first[k] .. c.link[c.group_first[k]], and its place in the
// list of all groups is c.list_base + k; the list's order is of no consequence.  A bucket that
// exceeds the capacity on its own is in no group.  Returns the largest bucket of the thread's warp.
// `most` and `capacity` may differ from one block to another, and with `other_count` groups of blocks that
// are `other` have a list of their own: group c.found + k of the block, k < c.found_other, is at c.other_base + k there.
__device__ __forceinline__ uint32_t cut_groups_of_block(GroupCut& c, int here, bool first_of_block, int block_end,
                                                        int longest, int most, uint32_t capacity, uint32_t* group_count,
                                                        uint32_t* other_count = nullptr, bool other = false) {
  const int tid = threadIdx.x;
  uint32_t load = 0;
  first_of_block = first_of_block && tid < here;
  block_end = min(here, block_end);
  int jump = kGroupSpan;
  if (tid < here) {
    load = c.start[tid + 1] - c.start[tid];
    int lo = tid + 1, hi = min(block_end, tid + most);  // the last end with start[end] - start[tid] <= capacity
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (c.start[mid] - c.start[tid] <= capacity) lo = mid; else hi = mid - 1;
    }
    c.link[tid] = static_cast<uint16_t>(lo);
    jump = lo < block_end ? lo : kGroupSpan;  // leaves its aligned block: no link
  }
  c.is_first[tid] = first_of_block;
  if (tid == 0) c.is_first[kGroupSpan] = 0;
  // The groups' first buckets: those reached from the blocks' first buckets along the
  // links, 2^k links at a time in round k.
  for (int hops = 1; hops < longest; hops <<= 1) {
    c.jumps[tid] = static_cast<uint16_t>(jump);
    if (tid == 0) c.jumps[kGroupSpan] = kGroupSpan;
    __syncthreads();
    const bool pass_on = c.is_first[tid];
    const int to = jump;
    jump = c.jumps[jump];
    __syncthreads();
    if (pass_on) c.is_first[to] = 1;
  }
  __syncthreads();
  if (tid < here && load > capacity) c.is_first[tid] = 0;  // too large for a group
  if (tid >= here) c.is_first[tid] = 0;
  const uint32_t mine = c.is_first[tid];
  // Both kinds in one scan, half a word each.
  const uint32_t place = block_exclusive_scan(mine << (other ? 16 : 0), c.warp_sum, &c.found);
  const uint32_t found = c.found & 0xffffu, found_other = c.found >> 16;
  if (mine) c.group_first[other ? found + (place >> 16) : place & 0xffffu] = static_cast<uint16_t>(tid);
  __syncthreads();
  if (tid == 0) {
    c.found = found;
    c.list_base = found ? atomicAdd(group_count, found) : 0u;
    c.found_other = found_other;
    if (found_other) c.other_base = atomicAdd(other_count, found_other);
  }
  __syncthreads();
  return __reduce_max_sync(0xffffffffu, load);
}

// A block takes kGroupSpan consecutive buckets.  Bucket starts: the records before bucket b are
// the records before it in every chunk, sum over c of run_begin[c][b] - (first record of c).
// The buckets are then cut into groups, and every group gets a table of where its records lie,
// two rows of table_row_words(chunks) words,
//   row 0: [c] first record of the group's run in chunk c; [chunks] first output slot of the
//          group; [chunks + 1], [chunks + 2] its buckets b0, b1
//   row 1: [c] records of the group in chunks before c; [chunks] records of the group.
// A bucket that exceeds the capacity on its own is in no group: finish_buckets takes it; one above
// `largest` cannot be finished at all and hands the call over before the scatter runs.
// Bound by latency: with a warp per group for its table and one thread following the links it
// took 22 us at 4 M particles (1250 buckets), with a chunk's loads one after the other 35 us at
// 64 M (16 chunks); now 6.5 and 19.
// `segments`: the sliced form, whose chunks begin at chunk_base[c] instead of c << chunk_log.
// ONE_CHUNK: `counts` are the buckets' counts, and the kernel does run_scan_kernel's work too: a block
// adds up what lies before its buckets for itself, and writes cursors and run_begin beside the
// bucket starts.  One launch less: 1 M particles without payload 44.9 -> 43.1 us per call, 4 M 96.2 -> 94.8,
// 1 M with payload 53.1 -> 52.5, 16 M without payload alike.
template <bool ONE_CHUNK>
__global__ void __launch_bounds__(kGroupSpan)
group_kernel(const uint32_t* counts, uint32_t n, uint32_t* cursor, uint32_t* run_begin, int buckets,
             int chunks, int chunk_log, const SliceSegments* __restrict__ segments, int group_shift,
             uint32_t capacity, uint32_t largest, uint32_t* __restrict__ bucket_start,
             uint32_t* __restrict__ tables, uint32_t* __restrict__ group_count, Header* __restrict__ hdr,
             bool behind) {
  // Behind a sort of a settled state the scatter kernel is chained too, and set up while these blocks hold
  // their multiprocessors its blocks would lie unevenly (17 M particles in random order, given up: 779 -> 645 us).
  if (!behind) chain_release();
  chain_wait();
  if (settled_before(hdr, behind)) return;
  // Up to kGroupStagedChunks chunks, [chunks][kGroupSpan + 1] each: the first record of every
  // run, and the records before the bucket in the chunks before c.
  extern __shared__ uint32_t staged[];
  __shared__ GroupCut cut;
  const int tid = threadIdx.x, lane = tid & 31;
  const int b0 = blockIdx.x * kGroupSpan;
  const int here = min(kGroupSpan, buckets - b0);
  const bool keep = chunks <= kGroupStagedChunks;
  uint32_t* earlier = staged + chunks * (kGroupSpan + 1);
  if (ONE_CHUNK) {
    uint32_t before = 0;
#pragma unroll 8
    for (int b = tid; b < b0; b += kGroupSpan) before += counts[b];
    if (tid == 0) cut.list_base = 0;
    const uint32_t mine = tid < here ? counts[b0 + tid] : 0u;
    before = __reduce_add_sync(0xffffffffu, before);
    const uint32_t inside = block_exclusive_scan(mine, cut.warp_sum, &cut.found);
    if (lane == 0 && before) atomicAdd(&cut.list_base, before);
    __syncthreads();
    const uint32_t start = cut.list_base + inside;
    if (tid < here) {
      cursor[b0 + tid] = start;
      run_begin[b0 + tid] = start;
    }
    if (tid <= here) cut.start[tid] = start;
    if (tid == here - 1) {
      cut.start[here] = start + mine;
      bucket_start[b0 + here] = start + mine;
      if (b0 + here == buckets) run_begin[buckets] = n;
    }
    if (tid < here) bucket_start[b0 + tid] = start;
    __syncthreads();
    for (int i = tid; i <= here; i += kGroupSpan) {
      staged[i] = cut.start[i];
      earlier[i] = 0;
    }
  }
  // Entry `here` (the end of the last bucket) is summed by the first thread as well.  The loads of
  // eight chunks are under way together.
  for (int i = tid; !ONE_CHUNK && i <= here; i += kGroupSpan) {
    uint32_t sum = 0;
    for (int c0 = 0; c0 < chunks; c0 += 8) {
      uint32_t s[8], base[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int c = min(c0 + k, chunks - 1);
        s[k] = run_begin[static_cast<size_t>(c) * buckets + b0 + i];
        base[k] = segments ? segments->chunk_base[c] : static_cast<uint32_t>(c) << chunk_log;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int c = c0 + k;
        if (c >= chunks) break;
        if (keep) {
          staged[c * (kGroupSpan + 1) + i] = s[k];
          earlier[c * (kGroupSpan + 1) + i] = sum;
        }
        sum += s[k] - base[k];
      }
    }
    cut.start[i] = sum;
    bucket_start[b0 + i] = sum;
  }
  __syncthreads();
  const uint32_t biggest = cut_groups_of_block(cut, here, (tid & ((1 << group_shift) - 1)) == 0, ((tid >> group_shift) + 1) << group_shift,
                                               1 << group_shift, 1 << group_shift, capacity, group_count);
  if (lane == 0 && biggest > 0) {
    atomicMax(&hdr->max_bucket, biggest);
    if (biggest > largest) hdr->use_standard = 1;
  }
  const uint32_t found = cut.found, list_base = cut.list_base;
  const uint32_t* start = cut.start;
  const uint16_t *link = cut.link, *group_first = cut.group_first;
  // The block's tables are one piece of memory: written word by word in order, whatever group and
  // chunk a word belongs to.
  const int row_words = table_row_words(chunks);
  uint32_t* table = tables + static_cast<size_t>(list_base) * 2 * row_words;
  if (keep) {
    const uint32_t words = found * 2 * row_words;
    for (uint32_t w = tid; w < words; w += kGroupSpan) {
      const uint32_t row = w / row_words, g = row >> 1;
      const int c = static_cast<int>(w - row * row_words);
      const int first = group_first[g], end = link[first];
      uint32_t value = 0;
      if (row & 1) {
        if (c < chunks) value = earlier[c * (kGroupSpan + 1) + end] - earlier[c * (kGroupSpan + 1) + first];
        else if (c == chunks) value = start[end] - start[first];
      } else {
        if (c < chunks) value = staged[c * (kGroupSpan + 1) + first];
        else if (c == chunks) value = start[first];
        else if (c == chunks + 1) value = static_cast<uint32_t>(b0 + first);
        else if (c == chunks + 2) value = static_cast<uint32_t>(b0 + end);
      }
      table[w] = value;
    }
  } else if (tid < static_cast<int>(found)) {
    const int first = group_first[tid], end = link[first];
    uint32_t* row0 = table + static_cast<size_t>(tid) * 2 * row_words;
    uint32_t* row1 = row0 + row_words;
    uint32_t offset = 0;
    for (int c = 0; c < chunks; ++c) {
      const uint32_t* row = run_begin + static_cast<size_t>(c) * buckets + b0;
      row0[c] = row[first];
      row1[c] = offset;
      offset += row[end] - row[first];
    }
    row0[chunks] = start[first];
    row0[chunks + 1] = static_cast<uint32_t>(b0 + first);
    row0[chunks + 2] = static_cast<uint32_t>(b0 + end);
    row1[chunks] = offset;
  }
}

// ------------------------------------------------------------------------
// Finish: a block sorts one group of buckets in shared memory and writes the output.
// ------------------------------------------------------------------------
constexpr uint32_t kBulkChunkBytes = 32768;  // bytes per bulk copy
constexpr uint32_t kBulkWaitLimit = 1u << 24;  // polls of the copy barrier
constexpr int kMaxSegments = 32;  // runs of cells an oversized bucket is cut into
constexpr int kMaxGroupBuckets = kGroupSpan;  // buckets in the aligned block a group may not leave
constexpr int kMaxChunks = 256;        // 2^30 particles in chunks of 2^22
constexpr int kTableRowWords = (kMaxChunks + 3 + 3) / 4 * 4;

// Two shapes of the finish kernel.  The small one runs two blocks per multiprocessor, so that
// one block's bulk copy and output stores overlap the other's ranking; it wants buckets of
// about a thousand records, which the count kernel's table can only offer up to about a
// hundred million particles.  Above that the large shape (one block per multiprocessor) runs.
template <int THREADS, int CAPACITY, int LOW_BITS, int RECORD_WORDS, int BLOCKS, int MAX_DROP>
struct FinishShape {
  static constexpr int kRecordWords = RECORD_WORDS;
  static constexpr int kBlocks = BLOCKS;                    // per multiprocessor
  static constexpr int kMaxDrop = MAX_DROP;                 // key bits left to the tie step, at most
  static constexpr int kMostIndexBits = RECORD_WORDS == kKeyRecordWords ? 7 : 0;  // see drop_for
  static constexpr int kThreads = THREADS;
  static constexpr int kCapacity = CAPACITY;                // records a block holds
  static constexpr int kItems = (CAPACITY + THREADS - 1) / THREADS;
  static constexpr int kLowBits = LOW_BITS;                 // key bits the counters resolve
  static constexpr int kHistWords = (1 << LOW_BITS) / 4;    // byte counters, 4 per word
  static constexpr int kWordsPerThread = kHistWords / THREADS;
  // A group spans at most this many cells: its low key (cell in group, shuffle bits) then has
  // at most LOW_BITS + MAX_DROP bits, of which the tie step may take MAX_DROP.
  static constexpr int kMaxCells = 1 << (LOW_BITS + MAX_DROP - kShuffleBits);
  // A run of cells cut from a bucket: few enough that every cell keeps 32 counters (5120 records on
  // 32 counters are 160 each; 16 wrap from some 3500 records on).
  static constexpr int kRunCells = 1 << (LOW_BITS + (MAX_DROP < 2 ? MAX_DROP : 2) - kShuffleBits);
  static constexpr uint32_t kLargestBucket = static_cast<uint32_t>(kMaxSegments) * CAPACITY;
  static_assert(kWordsPerThread % 8 == 0, "the counter scan reads eight words at a time");
  static_assert(kHistWords * 3 / 2 >= CAPACITY, "the tie step lays a word per record over the counters");
};
using FinishSmall = FinishShape<512, 2560, 14, kRecordWords, 2, 2>;
using FinishLarge = FinishShape<1024, 5120, 15, kRecordWords, 1, 2>;
// Calls without payload: 8-byte records and counters for half as many key bits leave room for
// three blocks of the large shape's capacity (with 2^15 counters, two blocks: 16 M particles 371
// us per call against 347, 4 M 116 against 111).  Three key bits may go to the tie step, so that
// sparse grids still have few buckets; indices must then stay below 2^29.
using FinishKeys = FinishShape<512, 5120, 14, kKeyRecordWords, 3, 3>;
constexpr int64_t kKeysMostParticles = int64_t{1} << 29;

template <class Shape>
struct __align__(128) FinishSmem {
  uint32_t raw[Shape::kCapacity * Shape::kRecordWords];  // the group's records as they lie in HBM
  union {
    struct {
      uint32_t hist[Shape::kHistWords];         // byte counter per low-key value
      uint16_t word_prefix[Shape::kHistWords];  // exclusive prefix of each counter word
    };
    uint32_t tie[Shape::kCapacity];  // what the tie step compares, when the counters are done with
  };
  uint16_t order[Shape::kCapacity];     // record held by each sorted slot
  uint32_t warp_sum[32];
  uint32_t total;
  uint32_t gave_up;
  uint32_t turn, groups, tasks;  // one-launch sort: what the block works on next; of how many
  unsigned long long barrier;    // mbarrier of the bulk copy
  uint32_t seg_begin[kMaxSegments + 1];  // oversized bucket: records before each run of cells
  uint16_t seg_first[kMaxSegments + 1];  // ... and the first cell of each run
  uint32_t fill;                         // ... and the records picked so far for the run at hand
};
// Behind the structure, in the same dynamic allocation: the tables of three consecutive
// groups, 2 * row_words words each (at most kTableRowWords per row).
constexpr size_t kSmallShapeTableBytes = 3 * 2 * 16 * sizeof(uint32_t);  // up to 13 chunks
static_assert(sizeof(FinishSmem<FinishLarge>) + 3 * 2 * kTableRowWords * sizeof(uint32_t) <=
                  227 * 1024, "finish kernel shared memory");
static_assert(2 * (sizeof(FinishSmem<FinishSmall>) + kSmallShapeTableBytes + 1024) <= 228 * 1024,
              "two small finish blocks must share a multiprocessor");
constexpr size_t kKeysShapeTableBytes = 3 * 2 * 20 * sizeof(uint32_t);  // up to 17 chunks
static_assert(3 * (sizeof(FinishSmem<FinishKeys>) + kKeysShapeTableBytes + 1024) <= 228 * 1024,
              "three finish blocks of a call without payload must share one");

template <class Shape>
__device__ __forceinline__ uint32_t* group_table(FinishSmem<Shape>& s, int q, int row_words) {
  return reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(&s) + sizeof(FinishSmem<Shape>)) +
         q * 2 * row_words;
}

__device__ __forceinline__ uint32_t byte_sum(uint32_t w) { return __dp4a(w, 0x01010101u, 0u); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Copies `bytes` (a multiple of 16, both addresses 16-byte aligned) from global
// to shared memory with the bulk-copy engine, in pieces of at most 32 KB; the
// bytes are counted on the mbarrier, which must already expect them.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes,
                                          unsigned long long* barrier) {
  const uint32_t bar = smem_addr(barrier);
  for (uint32_t done = 0; done < bytes; done += kBulkChunkBytes) {
    const uint32_t part = min(kBulkChunkBytes, bytes - done);
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_addr(static_cast<unsigned char*>(dst) + done)),
          "l"(static_cast<const unsigned char*>(src) + done), "r"(part), "r"(bar)
        : "memory");
  }
}

// Waits (bounded) for the phase `parity` of the copy barrier; false if it gave up: after
// kBulkWaitLimit polls, or after about two seconds on the global timer (a single poll may
// itself wait a while inside the hardware), whichever comes first.
__device__ __forceinline__ bool bulk_load_wait(unsigned long long* barrier, uint32_t parity) {
  const uint32_t bar = smem_addr(barrier);
  unsigned long long started = 0;
  for (uint32_t polls = 0; polls < kBulkWaitLimit; ++polls) {
    uint32_t ready;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ready) : "r"(bar), "r"(parity) : "memory");
    if (ready) return true;
    if ((polls & 1023u) == 1023u) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (started == 0) started = now;
      else if (now - started > 2000000000ull) return false;
    }
  }
  return false;
}

// Output arrays of the finish kernel.
struct FinishOut {
  uint32_t* keys;
  int32_t* index;
  int32_t* cell_counts;
  int32_t* cell_start;
  float* xs;
  float* ys;
  float* zs;
  float* vs;
  int64_t padded_sorted;
  int index_bits;  // every index is below 2^index_bits
};

// Key bits the byte counters must leave to the tie step for a set of `cells` cells; or, negative, how
// many of the index's highest bits they resolve besides the key.  With hundreds of particles to a
// cell a group has few cells and counters to spare, while every record shares its counter with
// others of its key; divided by index (which is what orders them) few do.  Calls without payload only:
// 4 M particles, 400 to a cell, 104.4 -> 98.3 us per call, 20 M with 200 466 -> 452; with payload, where the
// finish waits for other things, 50 M with 200 gain 0.7 % and thinner cells lose as much.
template <class Shape>
__device__ __forceinline__ int drop_for(int cells) {
  const int low_bits = (cells <= 1 ? 0 : 32 - __clz(cells - 1)) + kShuffleBits;
  return max(-Shape::kMostIndexBits, low_bits - Shape::kLowBits);
}
// Words of counters, four to a word: of a cell, and of `cells` of them.
__device__ __forceinline__ int cell_words_for(int drop) { return drop >= 0 ? 32 >> drop : 32 << -drop; }
__device__ __forceinline__ int counter_words(int cells, int drop) {
  return max(8, cells * cell_words_for(drop));
}

// Sorts the records at the first `places` places of s.raw (any order) and writes them to the
// output from slot `begin` on; `count` of the places hold a record, the others are passed over.
// `record_at(k, r, &key_index)`, called once by the thread that has place r as its k-th, tells
// whether there is one, and its key and index; it may first put the record there.
// The records belong to the cells first_cell ..
// first_cell + cells_here - 1 (at most Shape::kMaxCells).  The low key of a record is
// its key minus the key of the first cell's first shuffle value; the counters resolve
// all but its `drop` lowest bits, which the tie step orders together with the index, or, where
// drop is negative, all of it and -drop bits of the index.
// s.hist must be zero over the counters used; the call leaves it overwritten.
// Returns false if a byte counter wrapped (more than 255 records on one counter).
template <class Shape, class RecordAt>
__device__ __forceinline__ bool sort_placed(FinishSmem<Shape>& s, const FinishOut& out, int places, int count,
                                            uint32_t begin, int64_t first_cell, int cells_here,
                                            int drop, RecordAt record_at) {
  constexpr int kThreads = Shape::kThreads, kItems = Shape::kItems;
  constexpr int kWordsPerThread = Shape::kWordsPerThread;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t key_base = static_cast<uint32_t>(first_cell) << kShuffleBits;
  const int dropped = max(drop, 0), added = max(-drop, 0);
  const uint32_t drop_mask = (1u << dropped) - 1;
  const int index_shift = max(0, out.index_bits - added);
  const int cell_words = cell_words_for(drop);
  const int hist_words = counter_words(cells_here, drop);

  // Count the low key bits with byte-wide counters; the value an add returns
  // is the record's rank among the records of its counter.
  constexpr uint32_t kNoRecord = 0xffffffffu;
  uint32_t packed[kItems];  // counter id | rank << 16
  // What orders the records of one counter: dropped key bits, index.  (Read again from the
  // staged record where that is free of bank conflicts, kept in a register otherwise.)
  constexpr bool kKeep = Shape::kRecordWords != kKeyRecordWords;
  uint32_t mine[kKeep ? kItems : 1] = {};
  auto tie_word = [&](uint2 key_index) {
    return ((key_index.x & drop_mask) << (32 - Shape::kMaxDrop)) | key_index.y;
  };
  auto tie_word_of = [&](int k) {
    return kKeep ? mine[kKeep ? k : 0]
                 : tie_word(*reinterpret_cast<const uint2*>(
                       &s.raw[(tid + k * kThreads) * Shape::kRecordWords]));
  };
  auto count_records = [&](auto by_index) {
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int r = tid + k * kThreads;
      packed[k] = kNoRecord;
      if (kKeep) mine[kKeep ? k : 0] = 0;
      uint2 key_index;
      if (r < places && record_at(k, r, &key_index)) {
        const uint32_t low = decltype(by_index)::value
                                 ? ((key_index.x - key_base) << added) | (key_index.y >> index_shift)
                                 : (key_index.x - key_base) >> dropped;
        const int sh = 8 * (low & 3);
        const uint32_t old = atomicAdd(&s.hist[low >> 2], 1u << sh);
        packed[k] = low | (((old >> sh) & 0xffu) << 16);
        if (kKeep) mine[kKeep ? k : 0] = tie_word(key_index);
      }
    }
  };
  if (Shape::kMostIndexBits > 0 && added > 0) count_records(std::true_type());
  else count_records(std::false_type());
  __syncthreads();

  // Exclusive scan of the counters (8 words = 32 counters per thread, fetched
  // as two 128-bit loads so that neighbouring threads do not collide on banks).
  uint32_t local[kWordsPerThread];
  uint32_t sum = 0;
  {
#pragma unroll
    for (int j = 0; j < kWordsPerThread; j += 4) {
      uint4 a = make_uint4(0u, 0u, 0u, 0u);  // hist_words is a multiple of 4
      if (tid * kWordsPerThread + j < hist_words) a = *reinterpret_cast<const uint4*>(&s.hist[tid * kWordsPerThread + j]);
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        local[j + q] = sum;
        sum += byte_sum(w[q]);
      }
    }
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) s.warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kThreads / 32 ? s.warp_sum[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    s.warp_sum[lane] = wi - w;
    if (lane == 31) s.total = wi;
  }
  __syncthreads();
  const uint32_t thread_base = s.warp_sum[warp] + incl - sum;
#pragma unroll
  for (int j = 0; j < kWordsPerThread; j += 8)
    if (tid * kWordsPerThread + j < hist_words) {  // of eight words at its end four may lie past it: unused
      uint4 packed_prefix;
      packed_prefix.x = (thread_base + local[j]) | ((thread_base + local[j + 1]) << 16);
      packed_prefix.y = (thread_base + local[j + 2]) | ((thread_base + local[j + 3]) << 16);
      packed_prefix.z = (thread_base + local[j + 4]) | ((thread_base + local[j + 5]) << 16);
      packed_prefix.w = (thread_base + local[j + 6]) | ((thread_base + local[j + 7]) << 16);
      *reinterpret_cast<uint4*>(&s.word_prefix[tid * kWordsPerThread + j]) = packed_prefix;
    }
  // A byte counter that wrapped loses 256 from the total.
  const bool wrapped = s.total != static_cast<uint32_t>(count);
  __syncthreads();
  if (wrapped) return false;

  // Cell tables: every cell is cell_words words of consecutive counters.
  for (int c = tid; c < cells_here; c += kThreads) {
    const uint32_t lo = s.word_prefix[c * cell_words];
    const uint32_t hi = (c + 1) * cell_words < hist_words ? s.word_prefix[(c + 1) * cell_words]
                                                           : static_cast<uint32_t>(count);
    out.cell_start[first_cell + c] = static_cast<int32_t>(begin + lo);
    out.cell_counts[first_cell + c] = static_cast<int32_t>(hi - lo);
  }

  // Sorted slot of every record: start of its counter's run + arrival rank.  A
  // counter held by one record only (the usual case) is final at once.
  uint32_t run[kItems];  // run start | run length << 16, for records that share a counter
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int r = tid + k * kThreads;
    run[k] = 0;
    if (packed[k] != kNoRecord) {
      const uint32_t low = packed[k] & 0xffffu, rank = packed[k] >> 16;
      const uint32_t word = s.hist[low >> 2];
      const int sh = 8 * (low & 3);
      const uint32_t start = s.word_prefix[low >> 2] + byte_sum(word & ((1u << sh) - 1u));
      const uint32_t length = (word >> sh) & 0xffu;
      if (length > 1) run[k] = start | (length << 16);
      else s.order[start] = static_cast<uint16_t>(r);
    }
  }
  __syncthreads();

  // Records that share a counter must appear in ascending (dropped key bits,
  // original index): a record inside such a run goes to (run start + number of
  // smaller records in the run).  Indices stay below 2^(32 - kMaxDrop), so the dropped bits
  // ride above them in one word.  The words to compare are laid out run by run
  // over the counters, which nobody reads any more: a run is then a few
  // neighbouring words instead of as many records scattered over s.raw.
  uint32_t* tie = s.tie;
#pragma unroll
  for (int k = 0; k < kItems; ++k)
    if (run[k]) tie[(run[k] & 0xffffu) + (packed[k] >> 16)] = tie_word_of(k);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kItems; ++k)
    if (run[k]) {
      const uint32_t start = run[k] & 0xffffu, length = run[k] >> 16;
      const uint32_t word = tie_word_of(k);
      uint32_t smaller = 0;
      // Most runs are two or three records: four independent loads, then the rare rest.
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
        if (j < length) smaller += tie[start + j] < word;
      for (uint32_t j = 4; j < length; ++j) smaller += tie[start + j] < word;
      s.order[start + smaller] = static_cast<uint16_t>(tid + k * kThreads);
    }
  __syncthreads();

  // Coalesced output.
  if constexpr (Shape::kRecordWords == kKeyRecordWords) {
    for (int d = tid; d < count; d += kThreads) {
      const uint2 a = *reinterpret_cast<const uint2*>(&s.raw[s.order[d] * kKeyRecordWords]);
      const size_t o = static_cast<size_t>(begin) + d;
      __stcs(out.keys + o, a.x);
      __stcs(reinterpret_cast<uint32_t*>(out.index) + o, a.y);
    }
    __syncthreads();
    return true;
  }
  // A lane writes whole records, one word to each of the eight output arrays, so that a warp's store is
  // 128 bytes side by side and its address the same offset for all arrays.  Of every two
  // neighbouring lanes one reads its record's first half first and the other its second, so that a
  // quarter warp's eight halves fall on all banks.  Bound by instructions and the shared-memory pipe: with
  // two lanes to a record (half as many conflicts, twice the addresses, stores of two times 64 bytes) a call
  // took 2271 us at 64 M hypersonic, now 2234, and 3932 / 3844 at 128 M moved; 16 M and 1 M alike.
  {
    const bool odd = tid & 1;
    const uint32_t* const half = s.raw + (odd ? 4 : 0);
    const uint32_t* const other = s.raw + (odd ? 0 : 4);
    const bool positions = out.xs != nullptr, velocity = out.vs != nullptr;
    int next = tid < count ? s.order[tid] : 0;  // one round ahead of its use
    for (int d = tid; d < count; d += kThreads) {
      const int rec = next * kRecordWords;
      if (d + kThreads < count) next = s.order[d + kThreads];
      const uint4 a = *reinterpret_cast<const uint4*>(half + rec);
      const uint4 b = *reinterpret_cast<const uint4*>(other + rec);
      const uint32_t o = begin + d;
      __stcs(out.keys + o, odd ? b.x : a.x);
      __stcs(reinterpret_cast<uint32_t*>(out.index) + o, odd ? b.y : a.y);
      if (positions) {
        __stcs(reinterpret_cast<uint32_t*>(out.xs) + o, odd ? b.z : a.z);
        __stcs(reinterpret_cast<uint32_t*>(out.ys) + o, odd ? b.w : a.w);
        __stcs(reinterpret_cast<uint32_t*>(out.zs) + o, odd ? a.x : b.x);
      }
      if (velocity) {
        __stcs(reinterpret_cast<uint32_t*>(out.vs) + o, odd ? a.y : b.y);
        __stcs(reinterpret_cast<uint32_t*>(out.vs + out.padded_sorted) + o, odd ? a.z : b.z);
        __stcs(reinterpret_cast<uint32_t*>(out.vs + 2 * out.padded_sorted) + o, odd ? a.w : b.w);
      }
    }
  }
  __syncthreads();
  return true;
}

// The same for `count` records that all lie in s.raw.
template <class Shape>
__device__ __forceinline__ bool sort_staged(FinishSmem<Shape>& s, const FinishOut& out, int count,
                                            uint32_t begin, int64_t first_cell, int cells_here,
                                            int drop) {
  return sort_placed<Shape>(s, out, count, count, begin, first_cell, cells_here, drop,
                            [&](int, int r, uint2* key_index) {
    // Key and index in one access: it costs the same bank conflicts as the key alone.
    *key_index = *reinterpret_cast<const uint2*>(&s.raw[r * Shape::kRecordWords]);
    return true;
  });
}

// What the finish kernels need to find the records of a range of buckets.
struct RunTable {
  const uint32_t* records;
  const uint32_t* bucket_start;  // [buckets + 1]: records before each bucket, all chunks
  const uint32_t* run_begin;     // [chunks * buckets + 1]: first record of run (chunk, bucket)
  const uint32_t* tables;        // two rows of row_words words per group (group_kernel)
  const uint32_t* group_count;
  int row_words;
  int chunks;
  int buckets;
  int shift;                     // a bucket is 2^shift cells
  uint32_t* redo;                // room for the groups whose counters wrapped, or null
};

// The records of one bucket, run by run.
// `record_words`: from one record to the next; Shape's words of a record are its first.
template <class Shape>
struct BucketRecords {
  const RunTable& t;
  int b, record_words;
  template <class Each>
  __device__ __forceinline__ void runs(Each each) const {
    for (int c = 0; c < t.chunks; ++c) {
      const size_t entry = static_cast<size_t>(c) * t.buckets + b;
      const uint32_t start = t.run_begin[entry];
      each(start, t.run_begin[entry + 1] - start);
    }
  }
  template <class Use>
  __device__ __forceinline__ void keys(Use use) const {
    runs([&](uint32_t start, uint32_t length) {
      for (uint32_t base = 0; base < length; base += Shape::kThreads) {
        const bool valid = base + threadIdx.x < length;
        use(valid ? __ldcg(t.records + static_cast<size_t>(start + base + threadIdx.x) * record_words) : 0u, valid);
      }
    });
  }
  template <class Place>
  __device__ __forceinline__ void records(Place place) const {
    runs([&](uint32_t start, uint32_t length) {
      for (uint32_t i = threadIdx.x; i < length; i += Shape::kThreads) {
        const uint2* rec = reinterpret_cast<const uint2*>(t.records + static_cast<size_t>(start + i) * record_words);
        const uint2 lo = __ldcg(rec);
        uint2* to = reinterpret_cast<uint2*>(place(lo.x));
        if (!to) continue;
        to[0] = lo;
#pragma unroll
        for (int k = 1; k < Shape::kRecordWords / 2; ++k) to[k] = __ldcg(rec + k);
      }
    });
  }
};

// A bucket with more records than shared memory holds (a dense region: the
// bucket width is planned from the average load).  The block counts the
// bucket's records per cell, cuts the cells into up to kMaxSegments runs that
// fit, and for every run picks the run's records out of the bucket (which it
// reads from global memory once per run) and sorts them like a small group.
// Returns false if it cannot (a single cell larger than shared memory, too many
// runs, or a wrapped byte counter): the call then goes to the digit passes.
// `source`: where the bucket's records are.  source.keys(use) calls use(key, valid) for each of them, in
// whole warps; source.records(place) puts each record for whose key place(key) gives an address there.
// `after(first, count)`: what is left to do for these output slots when keys and indices stand.
template <class Shape, class Source, class After>
__device__ bool finish_large_bucket(FinishSmem<Shape>& s, const FinishOut& out, const Source& source,
                                    uint32_t begin, int64_t first_cell, int cells_here, After after) {
  constexpr int kThreads = Shape::kThreads, kCapacity = Shape::kCapacity;
  const int tid = threadIdx.x;
  static_assert(Shape::kMaxCells < Shape::kHistWords && Shape::kMaxCells <= 2 * kThreads, "cell counts");
  uint32_t* cell_count = s.hist;  // one word per cell; s.hist is free until a run is sorted
  for (int c = tid; c < cells_here; c += kThreads) cell_count[c] = 0;
  __syncthreads();
  // Per-cell counts: one pass over the keys of the bucket's records (lanes that agree share an
  // add: a bucket that comes here is crowded).
  source.keys([&](uint32_t key, bool valid) {
    bin_add(cell_count, (key >> kShuffleBits) - static_cast<uint32_t>(first_cell), valid);
  });
  __syncthreads();
  // Exclusive scan of the counts, two cells per thread, then one thread cuts the cells into runs
  // that fit, each as long as can be.  (Walking through the counts one by one took it as long as
  // all the rest.)
  {
    const int c0 = 2 * tid;
    const uint32_t n0 = c0 < cells_here ? cell_count[c0] : 0u, n1 = c0 + 1 < cells_here ? cell_count[c0 + 1] : 0u;
    const uint32_t before = block_exclusive_scan(n0 + n1, s.warp_sum, &s.total);
    if (c0 <= cells_here) cell_count[c0] = before;
    if (c0 + 1 <= cells_here) cell_count[c0 + 1] = before + n0;
    if (c0 + 2 == cells_here) cell_count[cells_here] = before + n0 + n1;
  }
  __syncthreads();
  if (tid == 0) {
    int segments = 0, c = 0;
    s.seg_first[0] = 0;
    s.seg_begin[0] = 0;
    while (c < cells_here && segments < kMaxSegments) {
      int lo = c, hi = min(cells_here, c + Shape::kRunCells);
      while (lo < hi) {  // the last end whose run still fits
        const int mid = (lo + hi + 1) >> 1;
        if (cell_count[mid] - cell_count[c] <= static_cast<uint32_t>(kCapacity)) lo = mid; else hi = mid - 1;
      }
      if (lo == c) break;  // a cell of its own does not fit
      c = lo;
      ++segments;
      s.seg_first[segments] = static_cast<uint16_t>(c);
      s.seg_begin[segments] = cell_count[c];
    }
    s.total = c == cells_here ? static_cast<uint32_t>(segments) : 0u;
  }
  __syncthreads();
  const int segments = static_cast<int>(s.total);
  __syncthreads();
  if (segments == 0) return false;
  for (int k = 0; k < segments; ++k) {
    const int c0 = s.seg_first[k], c1 = s.seg_first[k + 1];
    const uint32_t seg_begin = s.seg_begin[k];
    const int seg_count = static_cast<int>(s.seg_begin[k + 1] - seg_begin);
    const int drop = drop_for<Shape>(c1 - c0);
    // Zero the counters of this run and the fill cursor (cell_count is overwritten
    // from here on; the cuts above are already in seg_first / seg_begin).
    const int words = counter_words(c1 - c0, drop);
    for (int i = tid; i < words; i += kThreads) s.hist[i] = 0;
    if (tid == 0) s.fill = 0;
    __syncthreads();
    source.records([&](uint32_t key) -> uint32_t* {
      const int cell = static_cast<int>((key >> kShuffleBits) - static_cast<uint32_t>(first_cell));
      if (cell < c0 || cell >= c1) return nullptr;
      const uint32_t slot = atomicAdd(&s.fill, 1u);
      return slot < static_cast<uint32_t>(kCapacity) ? &s.raw[slot * Shape::kRecordWords] : nullptr;
    });
    __syncthreads();
    const bool consistent = s.fill == static_cast<uint32_t>(seg_count);
    __syncthreads();
    if (!consistent) return false;
    if (!sort_staged<Shape>(s, out, seg_count, begin + seg_begin, first_cell + c0, c1 - c0, drop))
      return false;
    after(begin + seg_begin, seg_count);
  }
  return true;
}

__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Starts the asynchronous copy of the table of group `g` (if there is one) into set `q`.
template <class Shape>
__device__ __forceinline__ void fetch_table(FinishSmem<Shape>& s, int q, const RunTable& t,
                                            uint32_t g, uint32_t groups) {
  const int pieces = 2 * t.row_words / 4;  // 16-byte pieces of the two rows
  if (g >= groups || static_cast<int>(threadIdx.x) >= pieces) return;
  const uint32_t* src = t.tables + static_cast<size_t>(g) * 2 * t.row_words + threadIdx.x * 4;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   smem_addr(group_table(s, q, t.row_words) + threadIdx.x * 4)), "l"(src) : "memory");
}

// Records of a call without payload: 8-byte asynchronous copies by all threads (a run may begin
// on any 8-byte boundary, which the bulk copies of touch_runs do not take).
template <class Shape>
__device__ __forceinline__ void fetch_key_records(FinishSmem<Shape>& s, int q, const RunTable& t) {
  const uint32_t* run_first = group_table(s, q, t.row_words);
  const uint32_t* run_offset = run_first + t.row_words;
  for (int c = 0; c < t.chunks; ++c) {
    const uint32_t offset = run_offset[c];
    const uint32_t length = min(run_offset[c + 1], static_cast<uint32_t>(Shape::kCapacity)) - offset;
    const uint32_t* src = t.records + static_cast<size_t>(run_first[c]) * kKeyRecordWords;
    for (uint32_t i = threadIdx.x; i < length; i += Shape::kThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                       smem_addr(&s.raw[(offset + i) * kKeyRecordWords])),
                   "l"(src + static_cast<size_t>(i) * kKeyRecordWords) : "memory");
  }
}

// Warp 0: the runs of the group whose table is in set `q`, one per chunk.  FETCH: bulk copies
// back to back into s.raw, counted on the barrier (lane 0 tells it first how many bytes to
// expect); otherwise only a request to bring the runs into L2, for the group after.
template <class Shape, bool FETCH>
__device__ __forceinline__ void touch_runs(FinishSmem<Shape>& s, int q, const RunTable& t) {
  const int lane = threadIdx.x & 31;
  const uint32_t* run_first = group_table(s, q, t.row_words);
  const uint32_t* run_offset = run_first + t.row_words;
  const uint32_t count = run_offset[t.chunks];
  if (count == 0) return;
  if (FETCH) {
    if (lane == 0) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                       smem_addr(&s.barrier)), "r"(count * kRecordWords * 4u) : "memory");
    }
    __syncwarp();
  }
  for (int c = lane; c < t.chunks; c += 32) {
    const uint32_t length = run_offset[c + 1] - run_offset[c];
    if (length == 0) continue;
    const uint32_t* src = t.records + static_cast<size_t>(run_first[c]) * kRecordWords;
    if (FETCH) {
      if (run_offset[c + 1] <= static_cast<uint32_t>(Shape::kCapacity))
        bulk_copy(s.raw + static_cast<size_t>(run_offset[c]) * kRecordWords, src,
                  length * kRecordWords * 4u, &s.barrier);
    } else {
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src),
                   "r"(length * kRecordWords * 4u) : "memory");
    }
  }
}

#include "settled_sort.cuh"

// `settled`: what the sort of a settled state before the kernel left, or NotSettled where there was none (in the tail kernel,
// with the arguments of such a sort 650,000 particles took 49.1 us instead of 48.4).
struct NotSettled {};

// A block works through groups blockIdx.x, blockIdx.x + gridDim.x, ... of the group list.
// What it needs to know about a group (where its runs lie) arrives two groups ahead by
// asynchronous copies; a group's records are asked into L2 while the group before it is
// sorted, and copied into shared memory as soon as that one's output is written.
// Behind a sort of a settled state it takes that sort's groups of dense regions.
template <class Shape, class Settled>
__global__ void __launch_bounds__(Shape::kThreads, Shape::kBlocks)
bucket_finish_kernel(RunTable t, int64_t n, const uint32_t* __restrict__ n_on_device,
                     int64_t num_cells, FinishOut out, Header* __restrict__ hdr, const __grid_constant__ Settled settled) {
  constexpr int kThreads = Shape::kThreads;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  chain_wait();
  if constexpr (std::is_same_v<Settled, SettledCall>) {
    if (settled_before(hdr, true)) {
      if (!finish_settled_dense<kThreads>(smem_raw, settled, blockIdx.x, gridDim.x)) hdr->use_standard = 1;
      return;
    }
  }
  const uint32_t groups = *t.group_count;
  if (handed_over(hdr)) return;
  FinishSmem<Shape>& s = *reinterpret_cast<FinishSmem<Shape>*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (blockIdx.x == 0 && tid == 0)
    out.cell_start[num_cells] = n_on_device ? static_cast<int32_t>(*n_on_device) : static_cast<int32_t>(n);
  const uint32_t stride = gridDim.x;
  uint32_t g = blockIdx.x;
  if (g >= groups) return;

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s.barrier)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s.gave_up = 0;
  }
  fetch_table<Shape>(s, 0, t, g, groups);
  fetch_table<Shape>(s, 1, t, g + stride, groups);
  copy_commit();
  copy_wait_all();
  __syncthreads();
  constexpr bool kBulk = Shape::kRecordWords == kRecordWords;
  if constexpr (!kBulk) {
    fetch_key_records<Shape>(s, 0, t);
    copy_commit();
  } else if (warp == 0) {
    touch_runs<Shape, true>(s, 0, t);
    if (g + stride < groups) touch_runs<Shape, false>(s, 1, t);
  }
  uint32_t parity = 0;

  for (int q = 0; g < groups; g += stride, q = q == 2 ? 0 : q + 1) {
    const int q1 = q == 2 ? 0 : q + 1, q2 = q1 == 2 ? 0 : q1 + 1;
    if constexpr (!kBulk) copy_wait_all();  // this group's records
    fetch_table<Shape>(s, q2, t, g + 2 * stride, groups);
    copy_commit();
    const uint32_t* row0 = group_table(s, q, t.row_words);
    const int count = static_cast<int>(row0[t.row_words + t.chunks]);
    const uint32_t begin = row0[t.chunks];
    const int b0 = static_cast<int>(row0[t.chunks + 1]), b1 = static_cast<int>(row0[t.chunks + 2]);
    const int64_t first_cell = static_cast<int64_t>(b0) << t.shift;
    const int cells_here = static_cast<int>(
        min(static_cast<long long>(b1 - b0) << t.shift, static_cast<long long>(num_cells - first_cell)));
    const int drop = drop_for<Shape>(cells_here);
    const int hist_words = counter_words(cells_here, drop);
    for (int i = tid; i < hist_words; i += kThreads) s.hist[i] = 0;
    if (kBulk && count > 0) {
      if (!bulk_load_wait(&s.barrier, parity)) s.gave_up = 1;
      parity ^= 1;
    }
    __syncthreads();
    if (s.gave_up) {  // the copy never landed: report and stop without touching the output
      if (tid == 0) atomicCAS(&hdr->error, 0, kErrBulkCopyTimeout);
      copy_wait_all();
      return;
    }
    if (!sort_staged<Shape>(s, out, count, begin, first_cell, cells_here, drop) && tid == 0) {
      if (t.redo) t.redo[atomicAdd(&hdr->redo_groups, 1u)] = g;
      else hdr->use_standard = 1;
    }
    // s.raw is free (sort_staged ended with a barrier): the next group's records, which L2
    // holds by now, can come in, and the group after it is asked into L2.
    copy_wait_all();
    __syncthreads();  // the table of group g + 2 * stride is visible
    if constexpr (!kBulk) {
      if (g + stride < groups) fetch_key_records<Shape>(s, q1, t);
      copy_commit();
    } else if (warp == 0) {
      if (g + stride < groups) touch_runs<Shape, true>(s, q1, t);
      if (g + 2 * stride < groups) touch_runs<Shape, false>(s, q2, t);
    }
  }
  chain_release();
}

// Buckets first, first + step, ... below `last` that hold at least `at_least` records, one by one:
// those the kernel above skipped, with more records than its shared memory holds, and those of a
// group whose counters wrapped.  False if one of them cannot be finished at all.
template <class Shape, class After>
__device__ bool finish_buckets(FinishSmem<Shape>& s, const RunTable& t, const FinishOut& out,
                               int64_t num_cells, int first, int last, int step, int at_least,
                               int record_words, After after) {
  for (int b = first; b < last; b += step) {
    const uint32_t begin = t.bucket_start[b], end = t.bucket_start[b + 1];
    const int count = static_cast<int>(end - begin);
    if (count < at_least) continue;
    const int64_t first_cell = static_cast<int64_t>(b) << t.shift;
    const int cells_here = static_cast<int>(
        min(static_cast<long long>(1) << t.shift, static_cast<long long>(num_cells - first_cell)));
    if (!finish_large_bucket<Shape>(s, out, BucketRecords<Shape>{t, b, record_words}, begin, first_cell, cells_here,
                                    after))
      return false;
  }
  return true;
}
template <class Shape>
__device__ bool finish_buckets(FinishSmem<Shape>& s, const RunTable& t, const FinishOut& out,
                               int64_t num_cells, int first, int last, int step, int at_least) {
  return finish_buckets<Shape>(s, t, out, num_cells, first, last, step, at_least, Shape::kRecordWords,
                               [](uint32_t, int) {});
}

// Behind the finish kernel of the multi-GPU form, which has no digit passes to hand over to.
template <class Shape>
__global__ void __launch_bounds__(Shape::kThreads, 1)
bucket_finish_large_kernel(RunTable t, int64_t num_cells, FinishOut out,
                           Header* __restrict__ hdr, uint32_t capacity) {
  chain_begin();
  if (handed_over(hdr) || hdr->max_bucket <= capacity) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (!finish_buckets<Shape>(*reinterpret_cast<FinishSmem<Shape>*>(smem_raw), t, out, num_cells,
                             blockIdx.x, t.buckets, gridDim.x, capacity + 1) &&
      threadIdx.x == 0)
    hdr->use_standard = 1;
}

// Behind the finish kernel of an ordinary call: the oversized buckets (of the sort of a settled state those that its
// dense groups do not hold) and the groups whose counters
// wrapped (calls without payload, whose sparse groups have 16 counters per cell), then, when the call was
// handed over, the whole digit-pass sort.  Usually there is nothing to do and every block returns
// after a look at the header.  What bounds it is then the launch itself: as the separate kernels
// it replaces (the oversized buckets, a clear, the keys, up to four digit passes, two table
// kernels and the payload gather, each returning at once) the same look cost 13-17 us of every
// call on the device and 11 launches on the host.
// Blocks per multiprocessor, fewer of them where there is little to do.
template <class Shape>
constexpr int kTailBlocks = Shape::kThreads <= 512 ? 2 : 1;
template <class Shape, class Settled>
__global__ void __launch_bounds__(Shape::kThreads, kTailBlocks<Shape>)
bucket_tail_kernel(RunTable t, int64_t num_cells, FinishOut out, Header* hdr, uint32_t capacity,
                   DigitPassArgs digits, const __grid_constant__ Settled settled) {
  constexpr bool kBehind = std::is_same_v<Settled, SettledCall>;
  chain_wait();
  const bool is_settled = settled_before(hdr, kBehind);
  const bool all_done = is_settled ? hdr->settle_large == 0 : hdr->max_bucket <= capacity && hdr->redo_groups == 0;
  if (!handed_over(hdr) && all_done) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const uint32_t items = gridDim.x;
  run_phases(hdr, items, 1 + digit_phases(digits), [&](uint32_t phase, uint32_t item) {
    const bool standard = handed_over(hdr);
    if (phase > 0)
      return standard && digit_phase<Shape::kThreads>(
                             digits, *reinterpret_cast<PassSmem<Shape::kThreads>*>(smem_raw), hdr,
                             phase - 1, item, items);
    // A block that comes late may see another block's hand-over and skip its buckets: the digit
    // passes then write everything.
    FinishSmem<Shape>& s = *reinterpret_cast<FinishSmem<Shape>*>(smem_raw);
    if constexpr (kBehind) {
      if (is_settled) {
        static_assert(Shape::kThreads == SettledWide::kThreads, "one block size");
        bool good = standard || finish_settled_groups(*reinterpret_cast<SettledSmem<SettledWide>*>(smem_raw), settled.args,
                                                      settled.out, settled.args.wide_tables, item, hdr->aux_counter[5], items,
                                                      threadIdx.x, BlockBarrier{});
        __syncthreads();
        good = good && (standard || finish_settled_large<Shape>(s, settled.args, settled.out, item, items));
        if (!good && threadIdx.x == 0) atomicExch(&hdr->use_standard, 1);
        return true;
      }
    }
    bool good = standard || finish_buckets<Shape>(s, t, out, num_cells, item, t.buckets, items, capacity + 1);
    for (uint32_t r = item; !standard && good && r < hdr->redo_groups; r += items) {
      const uint32_t* row0 = t.tables + static_cast<size_t>(t.redo[r]) * 2 * t.row_words;
      good = finish_buckets<Shape>(s, t, out, num_cells, row0[t.chunks + 1], row0[t.chunks + 2], 1, 0);
    }
    if (!good && threadIdx.x == 0) atomicExch(&hdr->use_standard, 1);
    return true;
  });
}

// ------------------------------------------------------------------------
// Small calls: the whole sort in one launch.
// ------------------------------------------------------------------------
// Up to here a call's time is the host's enqueueing of kernels and the latency of each; the work
// itself is a few microseconds.  A block takes one tile of at most kSmallItems particles per
// thread and keeps it in registers: it ranks the particles in their buckets (shared memory),
// reserves each bucket's places with one add per tile, and, when all tiles are counted, scans the
// bucket totals for itself and stores the records.  When all are stored the blocks finish the
// groups, and behind that the few calls that need it run the digit passes.
// On the device, as a memset and some twenty kernels / as a memset and this one: 200,003 particles
// with payload 44.6 / 27.5 us, 600,000 76 / 35; 5000 without payload take 13.  (Behind clear_kernel
// instead of a memset one to three microseconds less.)
// Usually all blocks run at once.  When they do not (something else holds multiprocessors), those
// that run count the tiles of those that don't, after kHelpAfterNs: a block waits for work that
// running blocks have taken on, and for nothing else.
constexpr int kSmallThreads = 512;
constexpr int kSmallItems = 4;
constexpr int kSmallMostBuckets = 2048;
// Buckets that are finished one by one are sorted by key and index only, whatever the call: the
// shape of calls without payload holds 5120 such records where the small shape holds 2560 with
// payload.  A cell with more than 2560 particles would otherwise take the call to the digit passes.
using FinishApart = FinishKeys;
constexpr uint32_t kFailedTask = 1u << 16;  // in tasks_done, above the number of tasks
static_assert(2 * (kSmallMostBuckets + kMaxTiles) < kFailedTask, "two counts in a word");
constexpr unsigned long long kHelpAfterNs = 50000;  // launch skew of a full grid: a few us

struct SmallArgs {
  const float *x, *y, *z, *v;
  int64_t padded, n, num_cells;
  PushSpec push;
  AetherGrid grid;
  uint32_t k0, k1;
  int shift, buckets, group_shift, items;
  int tiles;           // of items * kSmallThreads particles; the last ones may be empty
  uint32_t window;     // output slots per group, about
  uint32_t* count;     // [buckets], zero
  uint32_t* start;     // [buckets + 1]
  uint2* groups;       // [buckets]
  uint32_t* records;
};

template <class Shape>
struct SmallTables {  // over the records of the finish
  uint32_t *place, *start;
  __device__ __forceinline__ explicit SmallTables(FinishSmem<Shape>& s)
      : place(s.raw), start(s.raw + kSmallMostBuckets) {
    static_assert(sizeof(s.raw) >= 2 * (kSmallMostBuckets + 4) * sizeof(uint32_t), "room for both");
  }
};

__device__ __forceinline__ bool claim_tile(Header* hdr, int tile) {
  const uint32_t bit = 1u << (tile & 31);
  return (atomicOr(&hdr->tile_claimed[tile >> 5], bit) & bit) == 0;
}

template <int RECORD_WORDS>
__device__ __forceinline__ void store_small_record(const SmallArgs& a, uint32_t slot, uint32_t key,
                                                   int64_t i, const float* f) {
  uint32_t* record = a.records + static_cast<size_t>(slot) * RECORD_WORDS;
  if constexpr (RECORD_WORDS == kKeyRecordWords)
    *reinterpret_cast<uint2*>(record) = make_uint2(key, static_cast<uint32_t>(i));
  else
    store_record(record, key, static_cast<uint32_t>(i), f[0], f[1], f[2], f[3], f[4], f[5]);
}

// Particle i's values behind the fused move stage, and its cell.
__device__ __forceinline__ uint32_t small_cell(const SmallArgs& a, float* f) {
  if (a.push.enabled) {
#pragma unroll
    for (int c = 0; c < 3; ++c) push_axis(f[c], f[3 + c], a.push.dt, a.push.lo[c], a.push.hi[c]);
  }
  return cell_of(f[0], f[1], f[2], a.grid);
}
__device__ __forceinline__ void load_small(const SmallArgs& a, int64_t i, bool ok, float* f) {
  f[0] = ok ? a.x[i] : 0.f;
  f[1] = ok ? a.y[i] : 0.f;
  f[2] = ok ? a.z[i] : 0.f;
  f[3] = ok && a.v ? a.v[i] : 0.f;
  f[4] = ok && a.v ? a.v[a.padded + i] : 0.f;
  f[5] = ok && a.v ? a.v[2 * a.padded + i] : 0.f;
}

// The payload of output slots whose indices this very thread has written (sort_staged deals the
// slots out alike), from the inputs.
__device__ __forceinline__ void gather_small(const SmallArgs& a, const FinishOut& out, uint32_t from, int count) {
  for (int d = threadIdx.x; d < count; d += kSmallThreads) {
    const size_t o = static_cast<size_t>(from) + d;
    float f[6];
    load_small(a, out.index[o], true, f);
    small_cell(a, f);
    out.xs[o] = f[0];
    out.ys[o] = f[1];
    out.zs[o] = f[2];
    if (out.vs) {
      out.vs[o] = f[3];
      out.vs[out.padded_sorted + o] = f[4];
      out.vs[2 * out.padded_sorted + o] = f[5];
    }
  }
}

// One add per bucket and tile: a tile's counts become its first places in the buckets.
__device__ __forceinline__ void reserve_places(const SmallArgs& a, uint32_t* place) {
  for (int b = threadIdx.x; b < a.buckets; b += kSmallThreads) {
    const uint32_t c = place[b];
    if (c) place[b] = atomicAdd(&a.count[b], c);
  }
  __syncthreads();
}

// Bucket starts from the bucket totals; returns the largest total this thread has seen.
template <class Shape>
__device__ __forceinline__ uint32_t scan_totals(const SmallArgs& a, FinishSmem<Shape>& s) {
  uint32_t* start = SmallTables<Shape>(s).start;
  const int tid = threadIdx.x;
  uint32_t carry = 0, biggest = 0;
  for (int base = 0; base < a.buckets; base += kSmallThreads * 4) {
    uint32_t c[4], sum = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int b = base + tid * 4 + k;
      c[k] = b < a.buckets ? __ldcg(a.count + b) : 0u;
      sum += c[k];
      biggest = max(biggest, c[k]);
    }
    uint32_t before = carry + block_exclusive_scan(sum, s.warp_sum, &s.total);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int b = base + tid * 4 + k;
      if (b < a.buckets) start[b] = before;
      before += c[k];
    }
    carry += s.total;
    __syncthreads();  // the scan's scratch is used again
  }
  if (tid == 0) start[a.buckets] = static_cast<uint32_t>(a.n);
  __syncthreads();
  return biggest;
}

// Groups: a bucket begins one where an aligned block of buckets begins, where it or the bucket
// before it has more than half a block's records, and where its start passes into the next
// window (at most half the capacity) of output slots; so a group never has more than the
// capacity.  With every tile goes a share of the buckets, with the first what is written once.
template <class Shape>
__device__ __forceinline__ void cut_groups(const SmallArgs& a, const FinishOut& out, Header* hdr,
                                           const uint32_t* start, uint32_t biggest, int tile) {
  constexpr uint32_t kHalf = Shape::kCapacity / 2;
  const int tid = threadIdx.x;
  auto begins = [&](int b) {
    return (b & ((1 << a.group_shift) - 1)) == 0 || start[b + 1] - start[b] > kHalf ||
           start[b] - start[b - 1] > kHalf || start[b] / a.window != start[b - 1] / a.window;
  };
  const int share = (a.buckets + a.tiles - 1) / a.tiles;
  const int share_end = min(a.buckets, (tile + 1) * share);
  for (int b = tile * share + tid; b < share_end; b += kSmallThreads) {
    if (!begins(b) || start[b + 1] - start[b] > static_cast<uint32_t>(Shape::kCapacity)) continue;
    int end = b + 1;
    while (end < a.buckets && !begins(end)) ++end;
    a.groups[atomicAdd(&hdr->groups, 1u)] = make_uint2(static_cast<uint32_t>(b), static_cast<uint32_t>(end));
  }
  if (tile == 0) {
    for (int b = tid; b <= a.buckets; b += kSmallThreads) a.start[b] = start[b];
    biggest = __reduce_max_sync(0xffffffffu, biggest);
    if ((tid & 31) == 0) {
      atomicMax(&hdr->max_bucket, biggest);
      if (biggest > FinishApart::kLargestBucket) atomicExch(&hdr->use_standard, 1);
    }
    if (tid == 0) out.cell_start[a.num_cells] = static_cast<int32_t>(a.n);
  }
}

// A block that waits for blocks which do not run: it counts their tiles.  A tile counted here is
// loose: nobody holds it in registers.  Its particles' places in their buckets are left in the
// array of indices, which the finish overwrites, and when all tiles are counted any block that
// comes this way stores it.
template <class Shape>
__device__ __noinline__ bool place_loose_tiles(const SmallArgs& a, const FinishOut& out, Header* hdr,
                                               FinishSmem<Shape>& s) {
  constexpr uint32_t kNone = 0xffffffffu, kTaken = 0xfffffffeu;
  const SmallTables<Shape> table(s);
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) {
      const int left = a.tiles - 1 - static_cast<int>(atomicAdd(&hdr->help_next, 1u));
      s.turn = left < 0 ? kNone : claim_tile(hdr, left) ? static_cast<uint32_t>(left) : kTaken;
    }
    for (int b = tid; b < a.buckets; b += kSmallThreads) table.place[b] = 0;
    __syncthreads();
    const uint32_t tile = s.turn;
    __syncthreads();
    if (tile == kNone) break;
    if (tile == kTaken) continue;
    const int64_t first = static_cast<int64_t>(tile) * a.items * kSmallThreads + tid;
    for (int k = 0; k < a.items; ++k) {
      const int64_t i = first + k * kSmallThreads;
      if (i >= a.n) break;
      float f[6];
      load_small(a, i, true, f);
      const uint32_t b = small_cell(a, f) >> a.shift;
      out.keys[i] = b;
      out.index[i] = static_cast<int32_t>(atomicAdd(&table.place[b], 1u));
    }
    __syncthreads();
    reserve_places(a, table.place);
    for (int k = 0; k < a.items; ++k) {
      const int64_t i = first + k * kSmallThreads;
      if (i < a.n) out.index[i] += static_cast<int32_t>(table.place[out.keys[i]]);
    }
    if (tid == 0) atomicOr(&hdr->tile_loose[tile >> 5], 1u << (tile & 31));
    arrive(&hdr->tiles_counted);
  }
  if (!wait_for(&hdr->tiles_counted, a.tiles, &hdr->error)) return false;
  bool scanned = false;
  uint32_t biggest = 0;
  for (int w = 0; w * 32 < a.tiles;) {
    if (tid == 0) {
      uint32_t got = kNone;
      for (uint32_t bits; got == kNone && (bits = ld_relaxed(&hdr->tile_loose[w])) != 0;) {
        const uint32_t bit = bits & (0u - bits);
        if (atomicAnd(&hdr->tile_loose[w], ~bit) & bit) got = w * 32 + __ffs(bit) - 1;
      }
      __threadfence();  // the tile's places were written before its bit
      s.turn = got;
    }
    __syncthreads();
    const uint32_t tile = s.turn;
    __syncthreads();
    if (tile == kNone) {
      ++w;
      continue;
    }
    if (!scanned) biggest = scan_totals<Shape>(a, s);
    scanned = true;
    const int64_t first = static_cast<int64_t>(tile) * a.items * kSmallThreads + tid;
    for (int k = 0; k < a.items; ++k) {
      const int64_t i = first + k * kSmallThreads;
      if (i >= a.n) break;
      float f[6];
      load_small(a, i, true, f);
      const uint32_t cell = small_cell(a, f);
      store_small_record<Shape::kRecordWords>(
          a, table.start[cell >> a.shift] + static_cast<uint32_t>(__ldcg(out.index + i)),
          make_key(cell, static_cast<uint32_t>(i), a.k0, a.k1), i, f);
    }
    cut_groups<Shape>(a, out, hdr, table.start, biggest, static_cast<int>(tile));
    arrive(&hdr->tiles_stored);
  }
  return true;
}

template <class Shape>
__global__ void __launch_bounds__(kSmallThreads, 2)
small_sort_kernel(const __grid_constant__ SmallArgs a, const __grid_constant__ FinishOut out,
                  DigitPassArgs digits, Header* hdr) {
  static_assert(Shape::kThreads == kSmallThreads && FinishApart::kThreads == kSmallThreads,
                "one block size for all phases");
  static_assert(sizeof(FinishSmem<FinishApart>) <= sizeof(FinishSmem<Shape>), "shared memory");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FinishSmem<Shape>& s = *reinterpret_cast<FinishSmem<Shape>*>(smem_raw);
  const SmallTables<Shape> table(s);
  const int tid = threadIdx.x;
  const int tile = blockIdx.x;
  const int64_t first = static_cast<int64_t>(tile) * a.items * kSmallThreads + tid;

  for (int b = tid; b < a.buckets; b += kSmallThreads) table.place[b] = 0;
  __syncthreads();
  float f[kSmallItems][6];
  uint32_t key[kSmallItems], rank[kSmallItems];
#pragma unroll
  for (int k = 0; k < kSmallItems; ++k) {
    const int64_t i = first + k * kSmallThreads;
    load_small(a, i, k < a.items && i < a.n, f[k]);
  }
  chain_wait();  // the header is zero; the inputs were there before the kernel that zeroes it began
  // A block that starts late finds its tile claimed by another and goes on without one.  The
  // block's first task of the finish is asked for here, long before it is needed.
  uint32_t claimed = 0xffffffffu, next = 0;
  if (tid == 0) {
    claimed = atomicOr(&hdr->tile_claimed[tile >> 5], 1u << (tile & 31));
    next = atomicAdd(&hdr->task_next, 1u);
  }
  bool sharing = true;
#pragma unroll
  for (int k = 0; k < kSmallItems; ++k) {
    const int64_t i = first + k * kSmallThreads;
    const uint32_t cell = small_cell(a, f[k]);
    key[k] = make_key(cell, static_cast<uint32_t>(i), a.k0, a.k1);
    rank[k] = rank_in_tile(table.place, cell >> a.shift, k < a.items && i < a.n, sharing);
  }
  const bool holds = __syncthreads_or((claimed >> (tile & 31) & 1) == 0);
  if (holds) {
    reserve_places(a, table.place);
#pragma unroll
    for (int k = 0; k < kSmallItems; ++k) rank[k] += table.place[key[k] >> (kShuffleBits + a.shift)];
    arrive(&hdr->tiles_counted);
  }
  if (holds && wait_reaches(&hdr->tiles_counted, a.tiles, &hdr->error, kHelpAfterNs)) {
    const uint32_t biggest = scan_totals<Shape>(a, s);
#pragma unroll
    for (int k = 0; k < kSmallItems; ++k) {
      const int64_t i = first + k * kSmallThreads;
      if (k < a.items && i < a.n)
        store_small_record<Shape::kRecordWords>(
            a, table.start[key[k] >> (kShuffleBits + a.shift)] + rank[k], key[k], i, f[k]);
    }
    cut_groups<Shape>(a, out, hdr, table.start, biggest, tile);
    arrive(&hdr->tiles_stored);
  } else {
    if (holds) {  // lets its tile go before it helps
#pragma unroll
      for (int k = 0; k < kSmallItems; ++k) {
        const int64_t i = first + k * kSmallThreads;
        if (k < a.items && i < a.n) out.index[i] = static_cast<int32_t>(rank[k]);
      }
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        atomicOr(&hdr->tile_loose[tile >> 5], 1u << (tile & 31));
      }
    }
    if (!place_loose_tiles<Shape>(a, out, hdr, s)) return;
  }

  // The finish: tasks are the groups, and, where a bucket exceeds what a block holds, shares of
  // the buckets.  A block's next task is asked for while it works on one.
  if (tid == 0) s.turn = next;
  if (!wait_for(&hdr->tiles_stored, a.tiles, &hdr->error)) return;
  // One thread asks: thousands of warps that ask for one line queue there (606,208 particles: 2 us).
  if (tid == 0) {
    const uint32_t groups = ld_relaxed(&hdr->groups), max_bucket = ld_relaxed(&hdr->max_bucket);
    s.groups = groups;
    // No task at all where a bucket is beyond any block: the digit passes will write everything.
    s.tasks = max_bucket > FinishApart::kLargestBucket ? 0
              : max_bucket > static_cast<uint32_t>(Shape::kCapacity) ? groups + a.tiles : groups;
  }
  // Where there is no such group this reads what nobody uses.
  uint2 group = __ldcg(a.groups + min(s.turn, static_cast<uint32_t>(a.buckets) - 1));
  __syncthreads();
  const uint32_t groups = s.groups, tasks = s.tasks;
  uint32_t done = 0;  // tasks done here; failed ones count kFailedTask more
  for (;; ++done) {
    const uint32_t task = s.turn;
    if (task >= tasks) break;
    const RunTable t{a.records, a.start, a.start, nullptr, nullptr, 0, 1, a.buckets, a.shift, nullptr};
    int bucket = static_cast<int>(task - groups), last = a.buckets, step = a.tiles, at_least = Shape::kCapacity + 1;
    bool one_by_one = task >= groups;
    if (!one_by_one) {
      if (done > 0) group = __ldcg(a.groups + task);
      const uint32_t begin = __ldcg(a.start + group.x);
      const int count = static_cast<int>(__ldcg(a.start + group.y) - begin);
      const int64_t first_cell = static_cast<int64_t>(group.x) << a.shift;
      const int cells_here = static_cast<int>(
          min(static_cast<long long>(group.y - group.x) << a.shift, static_cast<long long>(a.num_cells - first_cell)));
      const int drop = drop_for<Shape>(cells_here);
      const int hist_words = counter_words(cells_here, drop);
      const uint2* from = reinterpret_cast<const uint2*>(a.records + static_cast<size_t>(begin) * Shape::kRecordWords);
      uint2* to = reinterpret_cast<uint2*>(s.raw);
#pragma unroll 8
      for (int i = tid; i < count * (Shape::kRecordWords / 2); i += kSmallThreads) to[i] = __ldcg(from + i);
      for (int i = tid; i < hist_words; i += kSmallThreads) s.hist[i] = 0;
      __syncthreads();
      if (tid == 0) next = atomicAdd(&hdr->task_next, 1u);
      one_by_one = !sort_staged<Shape>(s, out, count, begin, first_cell, cells_here, drop);
      bucket = group.x; last = group.y; step = 1; at_least = 0;
    } else if (tid == 0) {
      next = atomicAdd(&hdr->task_next, 1u);
    }
    if (one_by_one &&
        !finish_buckets<FinishApart>(
            *reinterpret_cast<FinishSmem<FinishApart>*>(smem_raw), t, out, a.num_cells, bucket, last, step,
            at_least, Shape::kRecordWords, [&](uint32_t from, int count) {
              if (Shape::kRecordWords != kKeyRecordWords) gather_small(a, out, from, count);
            }))
      done += kFailedTask;
    __syncthreads();
    if (tid == 0) s.turn = next;
    __syncthreads();
  }
  if (done >= kFailedTask && tid == 0) atomicExch(&hdr->use_standard, 1);
  chain_release();  // all blocks run by now: what is enqueued behind (the collisions of a step) may be set up
  arrive(&hdr->tasks_done, done);
  uint32_t seen = 0;
  if (!wait_for(&hdr->tasks_done, tasks, &hdr->error, kWaitLimitNs, kFailedTask - 1, &seen)) return;
  if (!__syncthreads_or(tid == 0 && seen >= kFailedTask) && tasks > 0) return;
  const uint32_t items = a.tiles;
  run_phases(hdr, items, digit_phases(digits), [&](uint32_t phase, uint32_t item) {
    return digit_phase<kSmallThreads>(digits, *reinterpret_cast<PassSmem<kSmallThreads>*>(smem_raw),
                                      hdr, phase, item, items);
  });
}

inline int index_bits_of(int64_t n) {
  int bits = 0;
  while ((int64_t{1} << bits) < n) ++bits;
  return bits;
}
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Above this many particles input in random order is scattered window by window, see scatter_span (20 M 649 -> 684 us per
// call, 33 M 1162 -> 1143, 50 M 1698 -> 1687, 64 M 2171 -> 2168, 75 M 2707 -> 2519, 100 M 3359 -> 3200).
constexpr int64_t kScatterWindowsFrom = int64_t{1} << 26;

// The chunk-major record layout: while a chunk is scattered its stores stay inside the
// chunk's region, which L2 serves faster than the whole record array; but every bucket gets
// one run per chunk, and short runs cost the scatter (partial lines) and the finish kernel
// (many small copies) more than the window saves.  Measured optimum on random input (us per call): 2^22 particles per chunk
// with 16 K buckets (64 M 2164 against 2271 with 2^23), 2^23 with 32 K or 64 K (100 M 3185 against 3298 with 2^22 and
// 3457 with 2^24, 128 M 4306 / 4486 / 4598, 256 M 9006 against 9422 with 2^24; also with 33 chunks, one more than the groups kernel
// keeps, 268,435,461 particles 9125 against 9535, 271 M 9225 against 9627), 2^24 beyond.  Smaller inputs take
// smaller chunks (fewer particles contend for a slot counter): best 2^20 at 4 M particles, 2^21 at 16 M.
inline int chunk_log_for(int64_t buckets, int64_t n) {
  if (n <= (int64_t{1} << 22)) return kChunkLog - 2;
  if (n <= (int64_t{1} << 24)) return kChunkLog - 1;
  return buckets <= (1 << 14) ? kChunkLog : buckets <= (1 << 16) ? kChunkLog + 1 : kChunkLog + 2;
}

// Particles from one round of a scatter block to its next (a power of two), where the input is in random order.  n / span
// windows of the record array are then written at a time, by blocks that started at different times: the slot counters
// they contend for are as many times as many.  With too many windows the lines that every bucket has open in each no
// longer stay in L2 until they are full: 128 bytes a bucket and window, best at 32 MB in all.  Every block has few
// rounds, and the next takes its place when it ends, which evens out that multiprocessors differ in speed (blocks that
// stay, and walk through the input in such an order: 128 M 4949 us per call, 256 M 11198; warps that draw their
// particles by ticket 4405, 9069).  us per call at log2 span: 100 M 22 3302, 23 3185, 24 3238; 128 M 22 4557, 24 4306, 25 4460; 256 M 24.6 10524, 25 9907, 26 9006,
// 27 9055.  (Before, two particles a thread and a span of 2.4 M whatever the size: 100 M 3359, 128 M 4695, 256 M 10392.)  Input
// in some order is better off that way: scattered window by window, 134 M moved by two cells take 4067 us against 3777.  Without payload a line takes sixteen records, and few windows are best: 100 M 24 2704, 25 2566,
// 26 2540, 27 2589; 150 M 25 4352, 26 4162, 27 4040; 200 M 25 6078, 26 5528, 27 5275 (before 2860, 4516, 6400).
int64_t scatter_span(int64_t n, int64_t buckets, bool keys_only) {
  const int64_t want = keys_only ? n / 2 : (n >> 9) * buckets / (1 << 9);
  int64_t span = int64_t{1} << 23;
  while (4 * span < want * 3) span *= 2;
  return span;
}

constexpr int kKeyChunkLog = 24;  // particles per chunk of a call without payload

struct BucketLayout {
  int chunk_log;
  int chunks;
  int64_t entries;  // chunks * buckets runs
  size_t count_off, start_off, cursor_off, run_begin_off, tables_off, records_off, total;
};

// Tables and records for `n` particles (or room for that many) in `chunks` chunks.
BucketLayout bucket_layout_of(int64_t n, int64_t buckets, int chunk_log, int chunks,
                              int record_words = kRecordWords) {
  BucketLayout l;
  l.chunk_log = chunk_log;
  l.chunks = chunks;
  l.entries = static_cast<int64_t>(l.chunks) * buckets;
  const size_t words = sizeof(uint32_t);
  l.count_off = sizeof(Header);  // zeroed per call together with the header
  l.start_off = align_up(l.count_off + l.entries * words, 256);  // zeroed up to here
  l.cursor_off = align_up(l.start_off + (buckets + 1) * words, 256);
  l.run_begin_off = align_up(l.cursor_off + l.entries * words, 256);
  l.tables_off = align_up(l.run_begin_off + (l.entries + 1) * words, 256);
  l.records_off = align_up(l.tables_off + buckets * 2 * table_row_words(l.chunks) * words, 256);
  l.total = align_up(l.records_off + static_cast<size_t>(n) * record_words * words, 256);
  return l;
}

BucketLayout bucket_layout(int64_t n, const BucketPlan& p) {
  const int64_t buckets = p.buckets;
  // Tiles split in shared memory write whole runs: no window has to be kept small for them.  Nor for 8-byte records
  // (scattered, with 2^24 particles to a chunk / 2^23, us per call: 32 K buckets 28 M 1029 / 1046, 50 M 1504 / 1568, 67 M 1915 / 2039, 101 M
  // 2629 / 2780, 135 M 3388 / 3630; 17 K buckets 20 M 673 / 687, 52 M 1424 / 1409, 101 M 2588 / 2809.  Below 2^26 either is ahead by up to 5 percent
  // at single sizes, 32 K buckets 16.9 M 818 / 784, 17 K buckets 36 M 1088 / 1034; 2^24 by one or two on average.)
  const int chunk_log = p.one_launch || p.tiled || p.keys_only ? kKeyChunkLog : chunk_log_for(buckets, n);
  const int chunks = static_cast<int>(
      std::max<int64_t>(1, (n + (int64_t{1} << chunk_log) - 1) >> chunk_log));
  return bucket_layout_of(n, buckets, chunk_log, chunks,
                          p.keys_only ? kKeyRecordWords : kRecordWords);
}

// Most buckets the small finish shape is planned for.  Beyond, the scatter pays more for the many
// small buckets than the finish kernel gains (us, buckets of 4096 records in the large shape / of
// 1024 in the small one): 64 M uniform count 138 / 203, scatter 1025 / 1409, finish 1018 / 858,
// call 2225 / 2507; 64 M hypersonic call 2245 / 2813; 128 M uniform count 296 / 884 (no table in
// shared memory), scatter 2415 / 3055, finish 2020 / 1723, call 4788 / 5713.  Up to the limit it
// gains: 32 M uniform call 1214 / 1127, 16 M 664 / 575.
constexpr int64_t kMaxSmallShapeBuckets = 32 * 1024;
int64_t g_small_shape_buckets = kMaxSmallShapeBuckets;  // tuning knob, see set_small_shape_buckets

// Blocks of the one-launch sort, and what it takes: a tile per resident block.
int small_call_most_blocks() { return std::min(2 * sm_count(), kMaxTiles); }
int64_t small_call_particles() {
  return static_cast<int64_t>(small_call_most_blocks()) * kSmallThreads * kSmallItems;
}
int small_call_blocks(int64_t n, int64_t buckets) {
  return static_cast<int>(std::max<int64_t>(
      1, std::min<int64_t>(small_call_most_blocks(), std::max((n + kSmallThreads - 1) / kSmallThreads, buckets / 8))));
}

// Up to where slots are reserved tile by tile.
constexpr int64_t kTiledMostParticles = 6 << 20;
constexpr int64_t kTiledMostBuckets = 8192;
// From here on tiles of 4096 particles, 1024 threads (against 2048, 512 threads, us per call: 2 M particles with 20 to a cell
// 86.1 / 85.6, 2.3 M 102.1 / 107.8, 3 M 119.5 / 123.1, 4 M 152.4 / 166.9; with 8 to a cell 91.1 / 93.4, 91.3 / 91.6, 110.1 / 113.4,
// 149.0 / 164.1).  Of nine sizes from 1.5 to 4 M at 4, 8, 20, 64 and 300 to a cell 3.2 M alone is slower for it, 4 percent
// at 4, 8 and 64 to a cell (126.6 / 121.7): not the number of rounds, which is the same either way.
constexpr int64_t kWideTilesFrom = 2300000;

// Largest bucket width 2^s, s <= max_shift, whose average load stays at or below `target`,
// with at least 2048 buckets (fewer make the slot counters of the scatter contend: measured
// at 1 M and 4 M particles, 2048 beats 1024, 4096 and 8192).
int shift_for(int64_t n, int64_t num_cells, int64_t target, int max_shift, int64_t fewest = 2048) {
  for (int s = max_shift; s > 0; --s) {
    const int64_t buckets = (num_cells + (int64_t{1} << s) - 1) >> s;
    if (n <= target * buckets && buckets >= fewest) return s;
  }
  return 0;
}

int log2_floor(int v) {
  int l = 0;
  while ((2 << l) <= v) ++l;
  return l;
}

}  // namespace

namespace {
// Records a group may hold: a finish block's capacity, or less where the groups would then not
// fill the rounds the blocks make (up to four; beyond, the last round matters little).  A quarter
// above an even share, so that whole buckets fit.
int64_t group_capacity_for(int64_t n, int capacity, int blocks_per_sm) {
  const int64_t blocks = static_cast<int64_t>(sm_count()) * blocks_per_sm;
  const int64_t rounds = std::max<int64_t>(1, (n + blocks * capacity - 1) / (blocks * capacity));
  if (rounds > 4) return capacity;
  return std::min<int64_t>(capacity, std::max<int64_t>(1024, n / (blocks * rounds) * 5 / 4));
}

// Output slots per group of the one-launch sort: an even share of a block, at most half of what
// a block holds.
uint32_t small_call_window(int64_t n, int64_t buckets, int capacity) {
  const int64_t blocks = small_call_blocks(n, buckets);
  return static_cast<uint32_t>(std::min<int64_t>(capacity / 2, std::max<int64_t>(64, (n + blocks - 1) / blocks)));
}

template <class Shape>
bool plan_one_launch(int64_t n, int64_t num_cells, BucketPlan* p) {
  if (n <= 0 || n > small_call_particles()) return false;
  // Buckets of half a window, so that groups are even.
  const int64_t target = small_call_window(n, 0, Shape::kCapacity) / 2;
  const int shift = shift_for(n, num_cells, target, log2_floor(Shape::kMaxCells), 1);
  const int64_t buckets = (num_cells + (int64_t{1} << shift) - 1) >> shift;
  if (buckets > kSmallMostBuckets || n > Shape::kCapacity * 2 / 5 * buckets) return false;
  p->shift = shift;
  p->buckets = buckets;
  p->usable = p->one_launch = true;
  return true;
}

// `tiled`: the call may use the one-launch sort or tile_scatter_kernel, to which few buckets are
// no burden.
BucketPlan plan_buckets_shape(int64_t n, int64_t num_cells, bool allow_small, bool tiled) {
  BucketPlan p;
  p.keys_only = p.tiled = p.one_launch = false;
  if (tiled && allow_small && plan_one_launch<FinishSmall>(n, num_cells, &p)) {
    p.small_blocks = true;
    if (p.buckets <= g_small_shape_buckets) return p;
    p.one_launch = false;
  }
  // The small finish shape (two blocks per multiprocessor) wants buckets well below its
  // capacity, so that the groups cut from them fill a block whatever the density does
  // inside a row of cells.
  p.small_blocks = true;
  if (tiled && allow_small && n <= kTiledMostParticles) {
    const int64_t target = std::min<int64_t>(
        1100, group_capacity_for(n, FinishSmall::kCapacity, FinishSmall::kBlocks) / 2);
    p.shift = shift_for(n, num_cells, target, log2_floor(FinishSmall::kMaxCells));
    p.buckets = (num_cells + (int64_t{1} << p.shift) - 1) >> p.shift;
    p.tiled = p.buckets <= kTiledMostBuckets;
    p.usable = p.tiled && n > 0 && n <= 1100 * p.buckets && p.buckets <= g_small_shape_buckets;
    if (p.usable) return p;
    p.tiled = false;
  }
  p.shift = shift_for(n, num_cells, 1100, log2_floor(FinishSmall::kMaxCells));
  p.buckets = (num_cells + (int64_t{1} << p.shift) - 1) >> p.shift;
  p.usable = allow_small && n > 0 && n <= 1100 * p.buckets && p.buckets <= g_small_shape_buckets;
  if (p.usable) return p;
  p.small_blocks = false;
  p.shift = shift_for(n, num_cells, 4160, log2_floor(FinishLarge::kMaxCells));
  p.buckets = (num_cells + (int64_t{1} << p.shift) - 1) >> p.shift;
  p.usable = n > 0 && n <= 4160 * p.buckets && p.buckets <= (int64_t{1} << 24);
  return p;
}
}  // namespace

BucketPlan plan_buckets(int64_t n, int64_t num_cells, bool keys_only) {
  if (!keys_only || n >= kKeysMostParticles) return plan_buckets_shape(n, num_cells, true, true);
  // Groups of a call without payload: a finish block's capacity, or less on small inputs so that
  // every block gets some; buckets of at most four fifths of that.
  BucketPlan p;
  p.keys_only = true;
  p.tiled = p.one_launch = false;
  p.small_blocks = false;
  if (plan_one_launch<FinishKeys>(n, num_cells, &p)) return p;
  const int64_t capacity = group_capacity_for(n, FinishKeys::kCapacity, FinishKeys::kBlocks);
  p.shift = shift_for(n, num_cells, capacity * 4 / 5 + 64, log2_floor(FinishKeys::kMaxCells), 1);
  p.buckets = (num_cells + (int64_t{1} << p.shift) - 1) >> p.shift;
  p.usable = n > 0 && n <= 4160 * p.buckets && p.buckets <= (int64_t{1} << 24);
  return p;
}

void set_small_shape_buckets(int64_t buckets) {
  g_small_shape_buckets = std::max<int64_t>(0, std::min<int64_t>(buckets, kMaxSmallShapeBuckets));
}

uint32_t bucket_group_capacity(int64_t n, const BucketPlan& p) {
  // A block's capacity, or less on small inputs so that every multiprocessor gets several groups.
  return static_cast<uint32_t>(group_capacity_for(
      n, p.keys_only ? FinishKeys::kCapacity : p.small_blocks ? FinishSmall::kCapacity
                                                              : FinishLarge::kCapacity,
      p.keys_only ? FinishKeys::kBlocks : p.small_blocks ? FinishSmall::kBlocks : FinishLarge::kBlocks));
}

size_t bucketed_workspace_bytes(int64_t n, int64_t num_cells, bool keys_only) {
  return bucket_layout(n, plan_buckets(n, num_cells, keys_only)).total;
}

namespace {

// Lets a kernel have `most` bytes of dynamic shared memory: the most that any call asks for, so
// that calls of different sizes from several threads set the same limit (with each call's own
// need as the limit, one thread could lower it between another's setting and launch).
template <class Kernel>
cudaError_t allow_shared(Kernel kernel, size_t most) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
}
constexpr size_t kMostCountTable = 200 * 1024;
constexpr size_t kMostGroupStage = 2 * kGroupStagedChunks * (kGroupSpan + 1) * sizeof(uint32_t);
constexpr size_t kMostSplitShared = 192 * 1024;
constexpr size_t kMostScanStage = (kStagedScanMax + 2 * (kFlatScanBlock + 1)) * sizeof(uint32_t);

// `counts`: of a call with one chunk, whose run_begin and cursors the kernel makes itself; or null.
cudaError_t launch_groups(cudaStream_t stream, const uint32_t* counts, int64_t n, uint32_t* cursor,
                          uint32_t* run_begin, int buckets, int chunks, int chunk_log, const SliceSegments* segments, int group_shift,
                          uint32_t capacity, uint32_t* start, uint32_t* tables, Header* hdr,
                          bool behind = false) {
  const size_t staged = chunks <= kGroupStagedChunks
                            ? 2 * static_cast<size_t>(chunks) * (kGroupSpan + 1) * sizeof(uint32_t) : 0;
  auto kernel = counts ? group_kernel<true> : group_kernel<false>;
  if (staged > 40 * 1024) {
    const cudaError_t e = allow_shared(kernel, kMostGroupStage);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(kernel, (buckets + kGroupSpan - 1) / kGroupSpan, kGroupSpan, staged, stream, counts,
                        n, cursor, run_begin, buckets, chunks, chunk_log, segments, group_shift, capacity,
                        FinishLarge::kLargestBucket, start, tables, &hdr->aux_counter[1], hdr, behind);
}

// Whether the kernels of a call that take long are chained (see chain_begin): without payload where tiles
// are split, and where slots are reserved tile by tile.  Without payload but with more buckets than a split
// takes, all chained / only the short ones: 75 M particles 2037 / 2009 us per call, 100 M 2984 / 2898, 200 M
// 6810 / 6470.  Those behind a sort of a settled state usually return at once (16.8 M
// 473 / 467 us, 64 M 1600 / 1593); where they do not, chaining costs nothing as long as each is let in only when
// the one before it ends.
bool heavy_chained(const BucketPlan& p, bool behind) {
  const bool split = p.keys_only && p.buckets <= kSplitMaxBuckets;
  return chained_launches() >= (behind || split || p.tiled ? 1 : 2);
}

template <class Shape, class Settled = NotSettled>
cudaError_t launch_finish(const RunTable& t, const SortArgs& a, const FinishOut& out, Header* hdr,
                          const uint32_t* n_on_device = nullptr, bool chained = false, const Settled& settled = {}) {
  const size_t table_bytes = 3 * 2 * static_cast<size_t>(t.row_words) * sizeof(uint32_t);
  if (std::is_same_v<Shape, FinishSmall> && table_bytes > kSmallShapeTableBytes)
    return cudaErrorInvalidValue;
  static_assert(std::is_same_v<Settled, NotSettled> ||
                    sizeof(SettledSmem<SettledDense>) * Shape::kThreads / SettledDense::kThreads <= sizeof(FinishSmem<Shape>),
                "shared memory");
  const int smem = static_cast<int>(sizeof(FinishSmem<Shape>) + table_bytes);
  auto kernel = bucket_finish_kernel<Shape, Settled>;
  cudaError_t e = allow_shared(kernel, sizeof(FinishSmem<Shape>) + 3 * 2 * kTableRowWords * sizeof(uint32_t));
  if (e != cudaSuccess) return e;
  return launch_chained_if(chained, kernel, std::min(t.buckets, sm_count() * Shape::kBlocks), Shape::kThreads, smem, a.stream,
                           t, a.n, n_on_device, a.num_cells, out, hdr, settled);
}

// Buckets in no group (more records than a group may hold) go to the large shape whatever
// the shape of the groups: a single cell may then hold up to its 5120 records.
cudaError_t launch_finish_large(const RunTable& t, const SortArgs& a, const FinishOut& out,
                                Header* hdr, uint32_t group_capacity) {
  constexpr int kSmem = static_cast<int>(sizeof(FinishSmem<FinishLarge>));
  cudaError_t e = allow_shared(bucket_finish_large_kernel<FinishLarge>, kSmem);
  if (e != cudaSuccess) return e;
  e = launch_chained<true>(bucket_finish_large_kernel<FinishLarge>, std::min(t.buckets, sm_count()),
                           FinishLarge::kThreads, kSmem, a.stream, t, a.num_cells, out, hdr,
                           group_capacity);
  return e != cudaSuccess ? e : cudaGetLastError();
}

int limited(int blocks, int most) { return most > 0 ? std::min(blocks, most) : blocks; }

template <class Shape, class Settled>
cudaError_t launch_tail(const RunTable& t, const SortArgs& a, const FinishOut& out, Header* hdr,
                        uint32_t group_capacity, const DigitPassArgs& digits, bool chained,
                        const Settled& settled) {
  constexpr int kSmem = static_cast<int>(std::max(sizeof(FinishSmem<Shape>), sizeof(PassSmem<Shape::kThreads>)));
  static_assert(std::is_same_v<Settled, NotSettled> ||
                    sizeof(SettledSmem<SettledWide>) <= kSmem, "shared memory");
  auto kernel = bucket_tail_kernel<Shape, Settled>;
  const cudaError_t e = allow_shared(kernel, kSmem);
  if (e != cudaSuccess) return e;
  const int blocks = static_cast<int>(std::max<int64_t>(
      1, std::min<int64_t>(sm_count() * kTailBlocks<Shape>, a.n / 2048)));
  return launch_chained_if(chained, kernel, limited(blocks, a.most_blocks), Shape::kThreads, kSmem, a.stream, t,
                           a.num_cells, out, hdr, group_capacity, digits, settled);
}

template <int THREADS>
cudaError_t launch_tile_scatter(const SortArgs& a, bool vec, uint32_t k0, uint32_t k1, int shift,
                                int buckets, int chunk_log, uint32_t* cursor, uint32_t* records,
                                Header* hdr, bool behind, bool chained) {
  constexpr int kTile = THREADS * 4;
  auto kernel = vec ? tile_scatter_kernel<true, THREADS> : tile_scatter_kernel<false, THREADS>;
  const int64_t tiles = (a.n + kTile - 1) / kTile;
  const int64_t blocks = behind ? std::min<int64_t>(tiles, sm_count() * (1024 / THREADS)) : tiles;
  return launch_chained_if(chained, kernel, static_cast<int>(blocks), THREADS,
                           static_cast<size_t>(buckets) * sizeof(uint32_t), a.stream, a.x, a.y, a.z,
                           a.velocity, a.padded, a.push, a.n, a.grid, k0, k1, shift, buckets, chunk_log,
                           cursor, records, hdr, behind);
}

template <int ITEMS, int THREADS>
cudaError_t launch_split(const SortArgs& a, bool vec, uint32_t k0, uint32_t k1, int shift, int buckets,
                         int chunk_log, uint32_t* cursor, uint32_t* records, Header* hdr, bool chained) {
  constexpr int kTile = THREADS * ITEMS;
  const size_t bytes = split_smem_bytes(kTile, buckets);
  const bool held = buckets <= kSplitHeld * THREADS;
  auto kernel = held ? (vec ? key_split_kernel<true, ITEMS, THREADS, true> : key_split_kernel<false, ITEMS, THREADS, true>)
                     : (vec ? key_split_kernel<true, ITEMS, THREADS, false> : key_split_kernel<false, ITEMS, THREADS, false>);
  static_assert(kTile * 8 + 2 * sizeof(uint32_t) * (kTile > 8192 ? kTile / 2 : kSplitMaxBuckets) <= kMostSplitShared,
                "shared memory");
  const cudaError_t e = allow_shared(kernel, kMostSplitShared);
  if (e != cudaSuccess) return e;
  // All blocks, and tiles as even as their rounds are (4 M particles: two of 6784 a block in place of two of 8192 for
  // some and one for the others); in one chunk, which a tile may not leave.  us per call, 8 to a cell, 1 M particles 41.8 -> 39.6, 1.6 M
  // 51.0 -> 45.9, 2.5 M 80.7 -> 74.3, 3 M 84.8 -> 77.7, 4 M 89.3 -> 87.3, 5 M 122.3 -> 114.1, 8 M 167 -> 163, 15 M 309 -> 304.
  const int64_t most = (THREADS <= 512 ? 2 : 1) * sm_count();
  const bool one_chunk = a.n <= int64_t{1} << chunk_log;
  const int64_t blocks = std::min<int64_t>(one_chunk ? (a.n + THREADS * 4 - 1) / (THREADS * 4) : (a.n + kTile - 1) / kTile, most);
  const int64_t rounds = (a.n + blocks * kTile - 1) / (blocks * kTile);
  const int64_t even = ((a.n + blocks * rounds - 1) / (blocks * rounds) + 127) / 128 * 128;
  const int tile = one_chunk ? static_cast<int>(std::min<int64_t>(even, kTile)) : kTile;
  return launch_chained_if(chained, kernel, static_cast<int>(blocks), THREADS, bytes, a.stream, a.x,
                              a.y, a.z, a.n, a.grid, k0, k1, shift, buckets, chunk_log, tile, cursor,
                              reinterpret_cast<uint2*>(records), hdr);
}

}  // namespace

namespace {
template <class Shape>
cudaError_t launch_small(const SortArgs& a, const BucketPlan& p, const BucketLayout& l,
                         const DigitPassArgs& digits) {
  constexpr int kSmem = static_cast<int>(std::max(sizeof(FinishSmem<Shape>), sizeof(PassSmem<kSmallThreads>)));
  static_assert(2 * (kSmem + 1024 + 64) <= 228 * 1024, "two blocks must share a multiprocessor");
  auto* base = static_cast<unsigned char*>(a.workspace);
  const cudaError_t e = allow_shared(small_sort_kernel<Shape>, kSmem);
  if (e != cudaSuccess) return e;
  const int blocks = small_call_blocks(a.n, p.buckets);
  SmallArgs s{};
  s.x = a.x; s.y = a.y; s.z = a.z; s.v = a.velocity;
  s.padded = a.padded; s.n = a.n; s.num_cells = a.num_cells;
  s.push = a.push;
  s.grid = a.grid;
  s.k0 = static_cast<uint32_t>(a.seed);
  s.k1 = static_cast<uint32_t>(a.seed >> 32);
  s.shift = p.shift;
  s.buckets = static_cast<int>(p.buckets);
  s.group_shift = std::max(0, log2_floor(Shape::kMaxCells) - p.shift);
  s.items = static_cast<int>((a.n + static_cast<int64_t>(blocks) * kSmallThreads - 1) /
                             (static_cast<int64_t>(blocks) * kSmallThreads));
  s.tiles = blocks;
  s.window = small_call_window(a.n, p.buckets, Shape::kCapacity);
  s.count = reinterpret_cast<uint32_t*>(base + l.count_off);
  s.start = reinterpret_cast<uint32_t*>(base + l.start_off);
  s.groups = reinterpret_cast<uint2*>(base + l.tables_off);
  s.records = reinterpret_cast<uint32_t*>(base + l.records_off);
  const FinishOut out{a.keys_out, a.index_out, a.cell_counts, a.cell_start, a.xs, a.ys, a.zs,
                      a.vs, a.padded_sorted, index_bits_of(a.n)};
  count_launches(1);
  return launch_chained(small_sort_kernel<Shape>, limited(blocks, a.most_blocks), kSmallThreads, kSmem, a.stream,
                        s, out, digits, reinterpret_cast<Header*>(base));
}
}  // namespace

namespace {
// From how many particles on a moved state is first tried as a settled one, where the general path
// would reserve its slots tile by tile, and where it would not.  us per call, general / settled / given up, five percent leaving
// their cell, or all: 1.6 M particles 72 / 68 / 91, 4 M 157 / 119 / 176, 6 M 216 / 159 / 240 (tiles); 8 M 253 / 208 / 286,
// 12.5 M 370 / 297 / 405, 15.5 M 448 / 358 / 490; 16.8 M 467 / 382 / 567, 30 M 805 / 637 / 925, 64 M 1794 / 1294 / 1965, 128 M
// 3555 / 2573 / 3890.  The second line was drawn with a finish that sorted whole records in shared memory (12.5 M 372 /
// 367, 16.8 M 479 / 460), where up to there a call had no more to gain than to lose by giving up (3 to 5 percent).  With the present finish it
// would gain 18 percent from 6.3 M on; the line has not been moved.
constexpr int64_t kSettledLeast = int64_t{3} << 19;
constexpr int64_t kSettledLeastUntiled = int64_t{1} << 24;
// Particles in a thousand that leave their bucket, above which the general path does the call (tiles; small finish blocks;
// large ones).  Up to there the settled sort is faster: us per call, movers in a thousand, settled / given up, 16.8 M 76 407 / 488;
// 64 M 129 1525 / 1835, 98 1475 / 1850; 128 M 98 2912 / 3631.  It would be beyond: without a limit, at 20 / 30 percent out of their cell 4 M
// 131 / 138 us against 168 given up, 16.8 M 447 / 484 against 494, 64 M 1536 / 1704 against 1841.  What the limits keep off is a call
// that fails late, when all the scan's lists are full (40 percent out of their cell: 209, 661, 2444 against 166, 504, 1888); from the
// limits to there is room for a sample that sees too few.  One block whose list is full costs nothing: 16.8 M 484 either way.
constexpr int64_t kMoversTiled = 180, kMoversSmall = 80, kMoversLarge = 140;

bool overlap(const void* a, size_t a_bytes, const void* b, size_t b_bytes) {
  const auto x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return x < y + b_bytes && y < x + a_bytes;
}

// Whether an output of the call lies over one of its inputs.  The general path reads the inputs for
// the last time before it writes the first output, so that such calls come out as if there
// were no overlap; the settled sort reads them while it writes.
bool outputs_over_inputs(const SortArgs& a) {
  const size_t row = static_cast<size_t>(a.n) * sizeof(float);
  const void* in[6] = {a.x, a.y, a.z, a.velocity, a.velocity + a.padded, a.velocity + 2 * a.padded};
  const void* out[8] = {a.keys_out, a.index_out, a.xs, a.ys, a.zs,
                        a.vs, a.vs + a.padded_sorted, a.vs + 2 * a.padded_sorted};
  for (const void* i : in) {
    for (const void* o : out)
      if (overlap(i, row, o, row)) return true;
    if (overlap(i, row, a.cell_counts, static_cast<size_t>(a.num_cells) * 4) ||
        overlap(i, row, a.cell_start, (static_cast<size_t>(a.num_cells) + 1) * 4))
      return true;
  }
  return false;
}

enum SettledKind { kSettledTeams, kSettledBlocks, kSettledSparse };  // the shape that sorts the usual groups
SettledKind settled_kind(int64_t n, int64_t num_cells) {
  if (n * SettledSparse::kMaxCells <= kSettledSparseMost * num_cells) return kSettledSparse;
  return n * SettledTeam::kMaxCells >= kSettledTeamLeast * num_cells && n <= kSettledTeamMostMean * num_cells ? kSettledTeams
                                                                                                              : kSettledBlocks;
}

// Lays the settled sort out in the `room` bytes at `base` (the general path's records, which that
// path writes after this one has given up); false if the call is not one for it.
bool settled_args(const SortArgs& a, const BucketPlan& p, unsigned char* base, size_t room, Header* hdr,
                  SettledArgs* out, size_t* zero_bytes) {
  if (!a.push.enabled || p.keys_only || !a.velocity || !a.vs || a.n < (p.tiled ? kSettledLeast : kSettledLeastUntiled) ||
      a.num_cells > (int64_t{1} << 25) - 1 || outputs_over_inputs(a))
    return false;
  SettledArgs s{};
  const SettledKind kind = settled_kind(a.n, a.num_cells);
  s.capacity = static_cast<uint32_t>(kind == kSettledTeams    ? SettledTeam::kCapacity
                                     : kind == kSettledBlocks ? SettledBlock::kCapacity : SettledSparse::kCapacity);
  s.most_cells = kind == kSettledTeams    ? SettledTeam::kMaxCells
                 : kind == kSettledBlocks ? SettledBlock::kMaxCells : SettledSparse::kMaxCells;
  s.shift = shift_for(a.n, a.num_cells, kind == kSettledTeams ? kSettledTeamTarget : kSettledBlockTarget, log2_floor(s.most_cells), 1);
  const int64_t buckets = (a.num_cells + (int64_t{1} << s.shift) - 1) >> s.shift;
  if (a.n > kSettledMostMean * buckets || buckets > a.n) return false;
  s.x = a.x; s.y = a.y; s.z = a.z; s.v = a.velocity;
  s.padded = a.padded; s.num_cells = a.num_cells;
  s.n = static_cast<int>(a.n);
  s.push = a.push;
  s.grid = a.grid;
  s.k0 = static_cast<uint32_t>(a.seed);
  s.k1 = static_cast<uint32_t>(a.seed >> 32);
  s.buckets = static_cast<int>(buckets);
  const int64_t most = static_cast<int64_t>(sm_count()) * 2;
  s.per_block = static_cast<int>(((a.n + most - 1) / most + kSettledRound - 1) / kSettledRound) * kSettledRound;
  s.scan_blocks = static_cast<int>((a.n + s.per_block - 1) / s.per_block);
  const int64_t in_last = a.n - static_cast<int64_t>(s.scan_blocks - 1) * s.per_block;
  const int64_t apart = s.per_block / kProbeSamples;
  const int64_t samples = static_cast<int64_t>(s.scan_blocks - 1) * kProbeSamples + (in_last + apart - 1) / apart;
  s.most_sampled = static_cast<uint32_t>(samples * (p.tiled ? kMoversTiled : p.small_blocks ? kMoversSmall : kMoversLarge) / 1000);
  s.most_movers = static_cast<uint32_t>(a.n / kMoverShare);
  s.hdr = hdr;
  s.vec_out = aligned16(a.keys_out) && aligned16(a.index_out) && aligned16(a.xs) && aligned16(a.ys) && aligned16(a.zs) &&
              aligned16(a.vs) && a.padded_sorted % 4 == 0;
  size_t used = 0;
  auto take = [&](int64_t words) {
    auto* at = reinterpret_cast<uint32_t*>(base + used);
    used = align_up(used + words * sizeof(uint32_t), 256);
    return at;
  };
  s.first = take(buckets);
  s.end = take(buckets);
  s.leavers = take(buckets);
  s.arrivals = take(buckets);
  *zero_bytes = used;
  s.keys = take(a.n);
  s.list_count = take(s.scan_blocks);
  s.cursor = take(buckets);
  s.sums = take((buckets + kSettledPart - 1) / kSettledPart * kSettledSums);
  s.tables = take(buckets * kSettledRowWords);
  s.dense_tables = take(buckets * kSettledRowWords);
  s.wide_tables = take((a.n / kSettledWideShare + 1) * kSettledRowWords);
  s.list = take(static_cast<int64_t>(s.scan_blocks) * (s.per_block / kListShare) * kRecordWords);
  s.arrived = take(static_cast<int64_t>(s.most_movers) * kRecordWords);
  *out = s;
  return used <= room;
}

template <class Shape>
cudaError_t launch_settled_finish(const SettledArgs& s, const FinishOut& out, cudaStream_t stream) {
  constexpr int kSmem = static_cast<int>(sizeof(SettledSmem<Shape>));
  const cudaError_t e = allow_shared(settled_finish_kernel<Shape>, kSmem);
  if (e != cudaSuccess) return e;
  return launch_chained(settled_finish_kernel<Shape>, sm_count() * Shape::kBlocks, Shape::kThreads, kSmem, stream, s, out);
}

// Enqueues the sort of a settled state; the general path's kernels follow it.
cudaError_t settled_sort(const SortArgs& a, const SettledArgs& s, size_t zero_bytes, const FinishOut& out) {
  constexpr int kScanSmem = static_cast<int>(sizeof(MoverQueue)) * (kSettledThreads / 32);
  const bool vec = aligned16(a.x) && aligned16(a.y) && aligned16(a.z) && aligned16(a.velocity) && a.padded % 4 == 0;
  const bool whole = a.grid.ix_offset == 0 && a.grid.nx_local == a.grid.nx;
  auto scan = vec ? (whole ? settled_scan_kernel<true, true> : settled_scan_kernel<true, false>)
                  : (whole ? settled_scan_kernel<false, true> : settled_scan_kernel<false, false>);
  cudaError_t e = allow_shared(scan, kScanSmem);
  if (e != cudaSuccess) return e;
  stage_begin(kStageBucketCount, a.stream);
  e = launch_chained(whole ? settled_probe_kernel<true> : settled_probe_kernel<false>, s.scan_blocks, kSettledThreads, 0,
                     a.stream, s, zero_bytes / sizeof(uint4));
  if (e == cudaSuccess) e = launch_chained(scan, s.scan_blocks, kSettledThreads, kScanSmem, a.stream, s);
  stage_end(kStageBucketCount, a.stream);
  stage_begin(kStageBucketScan, a.stream);
  if (e == cudaSuccess)
    e = launch_chained(settled_sums_kernel, (s.buckets + kSettledPart - 1) / kSettledPart, 1024, 0, a.stream, s);
  if (e == cudaSuccess)
    e = launch_chained(settled_groups_kernel, (s.buckets + kGroupSpan - 1) / kGroupSpan, kGroupSpan, 0, a.stream, s);
  stage_end(kStageBucketScan, a.stream);
  stage_begin(kStageBucketScatter, a.stream);
  if (e == cudaSuccess)
    e = launch_chained(settled_movers_kernel, s.scan_blocks, kSettledThreads, 0, a.stream, s);
  stage_end(kStageBucketScatter, a.stream);
  stage_begin(kStageBucketFinish, a.stream);
  const SettledKind kind = settled_kind(a.n, a.num_cells);
  const auto finish = kind == kSettledTeams    ? launch_settled_finish<SettledTeam>
                      : kind == kSettledBlocks ? launch_settled_finish<SettledBlock> : launch_settled_finish<SettledSparse>;
  if (e == cudaSuccess) e = finish(s, out, a.stream);
  count_launches(6);
  return e;
}

// Clears `bytes` at `base`, and the padding columns where they are the kernel's.  As many blocks as either takes: with
// those of the header and counts alone, two or three, 5001 particles with a million columns took 299 us (now 22), 1 M
// particles with a million 136 (60).
cudaError_t launch_clear(const SortArgs& a, void* base, size_t bytes) {
  const auto pieces = static_cast<int64_t>(bytes / sizeof(uint4));
  const int64_t columns = a.zero_padding ? a.padded_sorted - a.n : 0;
  const int blocks = static_cast<int>(std::min<int64_t>((std::max(pieces, columns) + 511) / 512, 2 * sm_count()));
  auto clear = a.zero_padding ? clear_kernel<true> : clear_kernel<false>;
  clear<<<blocks, 512, 0, a.stream>>>(static_cast<uint4*>(base), pieces, a.vs + a.n, a.padded_sorted, columns);
  count_launches(1);
  return cudaGetLastError();
}
}  // namespace

// What comes behind it is launched in the ordinary way (the memset of the digit passes, another clearing kernel), so that
// it is complete by then although it lets chained kernels in at once.
cudaError_t zero_padding_first(const SortArgs& a) { return launch_clear(a, nullptr, 0); }

// Enqueues the bucketed path.  When a bucket turns out too large for the finish
// kernel the device sets Header::use_standard, the kernels between return at once
// and the tail kernel runs the digit passes.
cudaError_t bucketed_sort(const SortArgs& a, const BucketPlan& p) {
  const BucketLayout l = bucket_layout(a.n, p);
  if (a.workspace_bytes < l.total || l.chunks > kMaxChunks) return cudaErrorInvalidValue;
  auto* base = static_cast<unsigned char*>(a.workspace);
  auto words_at = [&](size_t off) { return reinterpret_cast<uint32_t*>(base + off); };
  Header* hdr = reinterpret_cast<Header*>(base);
  uint32_t* count = words_at(l.count_off);
  uint32_t* start = words_at(l.start_off);
  uint32_t* cursor = words_at(l.cursor_off);
  uint32_t* run_begin = words_at(l.run_begin_off);
  uint32_t* tables = words_at(l.tables_off);
  uint32_t* records = words_at(l.records_off);
  DigitPassArgs digits;  // a workspace too small for them is refused before anything is enqueued
  cudaError_t e = digit_pass_args(a, &digits);
  if (e != cudaSuccess) return e;
  // Header and run counts.  An ordinary launch, which begins when all before it in the stream is done: the
  // kernels chained to it read the call's inputs before they wait for it.
  e = launch_clear(a, base, l.start_off);
  if (e != cudaSuccess) return e;
  if (p.one_launch) {
    stage_begin(kStageBucketFinish, a.stream);
    e = p.keys_only ? launch_small<FinishKeys>(a, p, l, digits) : launch_small<FinishSmall>(a, p, l, digits);
    stage_end(kStageBucketFinish, a.stream);
    return e;
  }
  const int buckets = static_cast<int>(p.buckets);
  const uint32_t k0 = static_cast<uint32_t>(a.seed), k1 = static_cast<uint32_t>(a.seed >> 32);
  const bool vec = aligned16(a.x) && aligned16(a.y) && aligned16(a.z) &&
                   (!a.velocity || (aligned16(a.velocity) && a.padded % 4 == 0));
  const FinishOut out{a.keys_out, a.index_out, a.cell_counts, a.cell_start, a.xs, a.ys, a.zs,
                      a.vs, a.padded_sorted, index_bits_of(a.n)};

  SettledCall settled{SettledArgs{}, out};
  size_t zero_bytes = 0;
  const bool behind = settled_args(a, p, base + l.records_off, l.total - l.records_off, hdr, &settled.args, &zero_bytes);
  if (behind) {
    e = settled_sort(a, settled.args, zero_bytes, out);
    if (e != cudaSuccess) return e;
  }
  const bool chained = heavy_chained(p, behind);
  // Behind a sort of a settled state the stages are that sort's, and the rest counts as its finish.
  auto begin_stage = [&](Stage stage) { if (!behind) stage_begin(stage, a.stream); };
  auto end_stage = [&](Stage stage) { if (!behind) stage_end(stage, a.stream); };

  uint32_t some_order;  // rounds of the count kernel's first warps that have seen neighbours in one bucket
  begin_stage(kStageBucketCount);
  {
    const size_t bytes32 = static_cast<size_t>(buckets) * sizeof(uint32_t);
    const size_t bytes16 = (static_cast<size_t>(buckets) + 1) / 2 * sizeof(uint32_t);
    const int table = bytes32 <= kMostCountTable ? kTableShared32
                      : bytes16 <= kMostCountTable ? kTableShared16 : kTableGlobal;
    const size_t table_bytes = table == kTableShared32 ? bytes32 : table == kTableShared16 ? bytes16 : 0;
    const bool wide = table_bytes > 96 * 1024;  // one 1024-thread block per SM holds the table
    const int threads = wide ? kCountThreadsWide : kCountThreads;
    const int blocks_per_sm = table == kTableGlobal ? 3 : wide ? 1 : table_bytes <= 64 * 1024 ? 3 : 2;
    // Equal shares, each a multiple of one block round (4 particles per thread) so that the
    // 16-byte loads stay aligned.
    const int64_t round = threads * 4;
    const int64_t most = static_cast<int64_t>(sm_count()) * blocks_per_sm;
    const int64_t per_block = std::max<int64_t>(kCountRounds, ((a.n + most - 1) / most + round - 1) / round) * round;
    const int grid = static_cast<int>((a.n + per_block - 1) / per_block);
    some_order = static_cast<uint32_t>(std::max<int64_t>(1, a.n / round / 2));
#define AETHER_COUNT_LAUNCH(TABLE, THREADS)                                                      \
  do {                                                                                            \
    auto kernel = vec ? bucket_count_kernel<TABLE, true, THREADS>                                 \
                      : bucket_count_kernel<TABLE, false, THREADS>;                               \
    if (table_bytes > 48 * 1024) {                                                                \
      e = allow_shared(kernel, kMostCountTable);                                                  \
      if (e != cudaSuccess) return e;                                                             \
    }                                                                                             \
    e = launch_chained_if(chained_launches() >= 1, kernel, grid, THREADS, table_bytes,  \
                          a.stream, a.x, a.y, a.z, a.velocity, a.padded, a.push, a.n, a.grid,     \
                          p.shift, buckets, l.chunk_log, per_block, count, hdr, behind);          \
    if (e != cudaSuccess) return e;                                                               \
  } while (0)
    if (table == kTableGlobal) AETHER_COUNT_LAUNCH(kTableGlobal, kCountThreads);
    else if (table == kTableShared16) AETHER_COUNT_LAUNCH(kTableShared16, kCountThreadsWide);
    else if (wide) AETHER_COUNT_LAUNCH(kTableShared32, kCountThreadsWide);
    else AETHER_COUNT_LAUNCH(kTableShared32, kCountThreads);
#undef AETHER_COUNT_LAUNCH
  }
  end_stage(kStageBucketCount);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;

  begin_stage(kStageBucketScan);
  const int max_cells = p.keys_only ? FinishKeys::kMaxCells
                        : p.small_blocks ? FinishSmall::kMaxCells : FinishLarge::kMaxCells;
  const uint32_t group_capacity = bucket_group_capacity(a.n, p);
  const int group_shift = std::min(log2_floor(kMaxGroupBuckets),
                                   std::max(0, log2_floor(max_cells) - p.shift));
  const dim3 scan_grid((buckets + kRunScanPart - 1) / kRunScanPart, l.chunks);
  const bool one_chunk = l.chunks == 1 && buckets <= kMostOneChunkBuckets;
  if (!one_chunk)
    e = launch_chained(run_scan_kernel, scan_grid, kRunScanThreads, 0, a.stream, count, buckets,
                       l.chunk_log, static_cast<uint32_t>(a.n), cursor, run_begin, hdr, behind);
  if (e == cudaSuccess)
    e = launch_groups(a.stream, one_chunk ? count : nullptr, a.n, cursor, run_begin, buckets, l.chunks,
                      l.chunk_log, nullptr, group_shift, group_capacity, start, tables, hdr, behind);
  if (e != cudaSuccess) return e;
  count_launches(one_chunk ? 1 : 2);
  end_stage(kStageBucketScan);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;

  begin_stage(kStageBucketScatter);
  if (p.keys_only && buckets <= kSplitMaxBuckets) {
    // Small inputs take small tiles, so that every block gets one, as long as one round is enough; with so many buckets that a
    // bucket's run in a tile of 8192 is shorter than four records (a 32-byte sector), large inputs
    // take tiles twice as large, one block per multiprocessor (whole call: 16 M particles, 4096
    // buckets 373 us against 386; 4 M, 1250 buckets 118 against 116).
    const int64_t sms = sm_count();
    const auto launch = buckets > 2048 && a.n >= sms * kSplitThreadsWide * 16
                            ? (buckets <= 8192 ? launch_split<16, kSplitThreadsWide>
                                               : launch_split<8, kSplitThreadsWide>)
                        : a.n > 2 * sms * kSplitThreads * 8 ? launch_split<16, kSplitThreads>
                        : a.n > 2 * sms * kSplitThreads * 4 ? launch_split<8, kSplitThreads>
                                                            : launch_split<4, kSplitThreads>;
    e = launch(a, vec, k0, k1, p.shift, buckets, l.chunk_log, cursor, records, hdr, chained);
    if (e != cudaSuccess) return e;
  } else if (p.tiled) {
    const auto launch = a.n >= kWideTilesFrom ? launch_tile_scatter<1024> : launch_tile_scatter<512>;
    e = launch(a, vec, k0, k1, p.shift, buckets, l.chunk_log, cursor, records, hdr, behind, chained);
    if (e != cudaSuccess) return e;
  } else {
    auto launch = [&](auto items, int64_t blocks, ScatterOnly only) {
      constexpr int kItems = decltype(items)::value;
      constexpr int kRound = kScatterThreads * kItems;
      auto kernel = p.keys_only ? (vec ? bucket_scatter_kernel<true, kItems, kKeyRecordWords>
                                       : bucket_scatter_kernel<false, kItems, kKeyRecordWords>)
                                : (vec ? bucket_scatter_kernel<true, kItems, kRecordWords>
                                       : bucket_scatter_kernel<false, kItems, kRecordWords>);
      const int grid = static_cast<int>(std::max<int64_t>(1, std::min((a.n + kRound - 1) / kRound, blocks)));
      return launch_chained_if(chained, kernel, grid, kScatterThreads, 0, a.stream, a.x, a.y, a.z,
                               a.velocity, a.padded, a.push, a.n, a.grid, k0, k1, p.shift, buckets, l.chunk_log,
                               cursor, records, hdr, only, some_order, behind);
    };
    using Two = std::integral_constant<int, 2>;
    using Four = std::integral_constant<int, 4>;
    // Behind a settled attempt one kernel for any order: a second that returns at once, too, costs settled states more than
    // windows gain those in random order (us per call without / with windows behind, settled 128 M 2680 / 2729, 256 M 7597 / 7732; random
    // 128 M 4900 / 4630, 256 M 9253 / 9385).
    const bool windows = !behind && a.n > kScatterWindowsFrom;
    e = launch(Two(), sm_count() * 16, windows ? kScatterOrdered : kScatterAny);
    if (e == cudaSuccess && windows) {
      e = launch(Four(), scatter_span(a.n, buckets, p.keys_only) / (kScatterThreads * 4), kScatterRandom);
      count_launches(1);
    }
    if (e != cudaSuccess) return e;
  }
  end_stage(kStageBucketScatter);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  count_launches(2);

  begin_stage(kStageBucketFinish);
  const RunTable t{records, start, run_begin, tables, &hdr->aux_counter[1],
                   table_row_words(l.chunks), l.chunks, buckets, p.shift, p.keys_only ? cursor : nullptr};
  e = p.keys_only      ? launch_finish<FinishKeys>(t, a, out, hdr, nullptr, chained)
      : p.small_blocks ? (behind ? launch_finish<FinishSmall>(t, a, out, hdr, nullptr, chained, settled)
                                 : launch_finish<FinishSmall>(t, a, out, hdr, nullptr, chained))
      : behind         ? launch_finish<FinishLarge>(t, a, out, hdr, nullptr, chained, settled)
                       : launch_finish<FinishLarge>(t, a, out, hdr, nullptr, chained);
  if (e == cudaSuccess)
    e = behind        ? launch_tail<FinishLarge>(t, a, out, hdr, group_capacity, digits, chained, settled)
        : p.keys_only ? launch_tail<FinishKeys>(t, a, out, hdr, group_capacity, digits, chained, NotSettled{})
                      : launch_tail<FinishLarge>(t, a, out, hdr, group_capacity, digits, chained, NotSettled{});
  stage_end(kStageBucketFinish, a.stream);
  count_launches(2);
  return e;
}

// ---- the segmented form: one chunk per slice of the sliced exchange ----

namespace {
// The small shape's shared memory has room for the tables of a dozen chunks only.
BucketPlan sliced_plan(int64_t plan_n, int64_t num_cells, int slices) {
  const bool tables_fit =
      3 * 2 * static_cast<size_t>(table_row_words(slices)) * sizeof(uint32_t) <= kSmallShapeTableBytes;
  return plan_buckets_shape(plan_n, num_cells, tables_fit, false);
}
}  // namespace

size_t sliced_sort_workspace_bytes(int64_t capacity, int64_t plan_n, int64_t num_cells, int slices) {
  const BucketPlan p = sliced_plan(plan_n, num_cells, slices);
  return bucket_layout_of(capacity, p.buckets, 0, slices).total;
}

namespace {
struct SlicedState {
  BucketPlan plan;
  BucketLayout layout;
  unsigned char* base;
  bool ok;
};
SlicedState sliced_state(const SortArgs& a, int64_t plan_n, int slices) {
  SlicedState st{};
  st.plan = sliced_plan(plan_n, a.num_cells, slices);
  st.layout = bucket_layout_of(a.n, st.plan.buckets, 0, slices);
  st.base = static_cast<unsigned char*>(a.workspace);
  st.ok = st.plan.usable && slices >= 1 && slices <= kMaxSlices && a.workspace &&
          a.workspace_bytes >= st.layout.total &&
          (reinterpret_cast<uintptr_t>(a.workspace) & 255) == 0;
  return st;
}
}  // namespace

cudaError_t sliced_sort_begin(const SortArgs& a, int64_t plan_n, int slices) {
  const SlicedState st = sliced_state(a, plan_n, slices);
  if (!st.ok) return cudaErrorInvalidValue;
  stage_reset();
  return cudaMemsetAsync(st.base, 0, st.layout.start_off, a.stream);  // header and run counts
}

cudaError_t sliced_sort_slice(const SortArgs& a, int64_t plan_n, const SliceSegments* segments,
                              int slices, int slice) {
  const SlicedState st = sliced_state(a, plan_n, slices);
  if (!st.ok || !segments || slice < 0 || slice >= slices) return cudaErrorInvalidValue;
  if (!a.x || !a.y || !a.z || !a.velocity || a.padded < a.n) return cudaErrorInvalidValue;
  const BucketLayout& l = st.layout;
  auto words_at = [&](size_t off) { return reinterpret_cast<uint32_t*>(st.base + off); };
  const int buckets = static_cast<int>(st.plan.buckets);
  uint32_t* row = words_at(l.count_off) + static_cast<size_t>(slice) * buckets;
  uint32_t* cursor_row = words_at(l.cursor_off) + static_cast<size_t>(slice) * buckets;
  uint32_t* run_begin_row = words_at(l.run_begin_off) + static_cast<size_t>(slice) * buckets;
  uint32_t* records = words_at(l.records_off);
  const bool vec = aligned16(a.x) && aligned16(a.y) && aligned16(a.z) && aligned16(a.velocity) &&
                   a.padded % 4 == 0;
  // Work units of a slice: its share of the planned particles, and one partial unit per source.
  const int64_t units = plan_n / slices / kSegmentUnit + kMaxWorld + 1;
  cudaError_t e = cudaSuccess;

  stage_begin(kStageBucketCount, a.stream);
  {
    const size_t table_bytes = static_cast<size_t>(buckets) * sizeof(uint32_t);
    const bool shared = table_bytes <= kMostCountTable;
    const bool wide = shared && table_bytes > 96 * 1024;
    const int per_sm = !shared ? 4 : wide ? 1 : table_bytes <= 48 * 1024 ? 4 : 2;
    const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(units, sm_count() * per_sm)));
    if (!shared) {
      bucket_count_segments_kernel<kTableGlobal, kCountThreads><<<grid, kCountThreads, 0, a.stream>>>(
          a.x, a.y, a.z, a.n, vec, segments, slice, a.grid, st.plan.shift, buckets, row);
    } else if (wide) {
      auto kernel = bucket_count_segments_kernel<kTableShared32, kCountThreadsWide>;
      e = allow_shared(kernel, kMostCountTable);
      if (e != cudaSuccess) return e;
      kernel<<<grid, kCountThreadsWide, table_bytes, a.stream>>>(
          a.x, a.y, a.z, a.n, vec, segments, slice, a.grid, st.plan.shift, buckets, row);
    } else {
      auto kernel = bucket_count_segments_kernel<kTableShared32, kCountThreads>;
      if (table_bytes > 48 * 1024) {
        e = allow_shared(kernel, kMostCountTable);
        if (e != cudaSuccess) return e;
      }
      kernel<<<grid, kCountThreads, table_bytes, a.stream>>>(
          a.x, a.y, a.z, a.n, vec, segments, slice, a.grid, st.plan.shift, buckets, row);
    }
  }
  stage_end(kStageBucketCount, a.stream);
  stage_begin(kStageBucketScan, a.stream);
  if (buckets <= kStagedScanMax) {
    const int per = (buckets + kFlatScanBlock - 1) / kFlatScanBlock;
    const size_t bytes = (static_cast<size_t>(buckets) + 2 * (buckets / per + 1)) * sizeof(uint32_t);
    if (bytes > 48 * 1024) {
      e = allow_shared(chunk_scan_kernel<true>, kMostScanStage);
      if (e != cudaSuccess) return e;
    }
    chunk_scan_kernel<true><<<1, kFlatScanBlock, bytes, a.stream>>>(row, buckets, segments, slice,
                                                                    cursor_row, run_begin_row);
  } else {
    chunk_scan_kernel<false><<<1, kFlatScanBlock, 0, a.stream>>>(row, buckets, segments, slice,
                                                                 cursor_row, run_begin_row);
  }
  stage_end(kStageBucketScan, a.stream);
  stage_begin(kStageBucketScatter, a.stream);
  {
    constexpr int kItems = 2;
    const int grid = static_cast<int>(std::max<int64_t>(
        1, std::min<int64_t>(units, sm_count() * (8 / kItems))));
    const uint32_t k0 = static_cast<uint32_t>(a.seed), k1 = static_cast<uint32_t>(a.seed >> 32);
    bucket_scatter_segments_kernel<kItems><<<grid, kScatterThreads, 0, a.stream>>>(
        a.x, a.y, a.z, a.velocity, a.padded, a.n, vec, segments, slice, a.grid, k0, k1,
        st.plan.shift, buckets, cursor_row, records);
  }
  stage_end(kStageBucketScatter, a.stream);
  count_launches(3);
  return cudaGetLastError();
}

cudaError_t sliced_sort_finish(const SortArgs& a, int64_t plan_n, const SliceSegments* segments,
                               int slices) {
  const SlicedState st = sliced_state(a, plan_n, slices);
  if (!st.ok || !segments) return cudaErrorInvalidValue;
  if (!a.keys_out || !a.index_out || !a.cell_counts || !a.cell_start) return cudaErrorInvalidValue;
  const BucketLayout& l = st.layout;
  const BucketPlan& p = st.plan;
  auto words_at = [&](size_t off) { return reinterpret_cast<uint32_t*>(st.base + off); };
  Header* hdr = reinterpret_cast<Header*>(st.base);
  const int buckets = static_cast<int>(p.buckets);
  uint32_t* start = words_at(l.start_off);
  uint32_t* run_begin = words_at(l.run_begin_off);
  uint32_t* tables = words_at(l.tables_off);
  uint32_t* records = words_at(l.records_off);
  const uint32_t* n_on_device = &segments->n;

  stage_begin(kStageBucketFinish, a.stream);
  const int max_cells = p.small_blocks ? FinishSmall::kMaxCells : FinishLarge::kMaxCells;
  const uint32_t group_capacity = bucket_group_capacity(plan_n, p);
  const int group_shift = std::min(log2_floor(kMaxGroupBuckets),
                                   std::max(0, log2_floor(max_cells) - p.shift));
  cudaError_t e = launch_groups(a.stream, nullptr, 0, nullptr, run_begin, buckets, l.chunks, 0, segments,
                                group_shift, group_capacity, start, tables, hdr);
  if (e != cudaSuccess) return e;
  count_launches(3);
  const FinishOut out{a.keys_out, a.index_out, a.cell_counts, a.cell_start, a.xs, a.ys, a.zs,
                      a.vs, a.padded_sorted, index_bits_of(a.n)};
  const RunTable t{records, start, run_begin, tables, &hdr->aux_counter[1],
                   table_row_words(l.chunks), l.chunks, buckets, p.shift, nullptr};
  e = p.small_blocks ? launch_finish<FinishSmall>(t, a, out, hdr, n_on_device)
                     : launch_finish<FinishLarge>(t, a, out, hdr, n_on_device);
  if (e == cudaSuccess) e = launch_finish_large(t, a, out, hdr, group_capacity);
  stage_end(kStageBucketFinish, a.stream);
  return e;
}

}  // namespace aether
