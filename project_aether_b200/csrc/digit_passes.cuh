// Device bodies of the digit passes, used by the kernels of the digit-pass path
// (sort_standard.cu: one launch per pass) and by the kernel behind the bucketed path
// (sort_bucketed.cu: all passes in one launch, for the calls the bucketed
// path hands over).  Buffers that one pass writes and the next one reads are plain
// pointers (no __restrict__): inside one launch they must not be read through the
// non-coherent cache.
#pragma once

#include "common.cuh"

namespace aether {

// ------------------------------------------------------------------------
// One Onesweep digit pass.
// ------------------------------------------------------------------------
constexpr int kPassTile = 6144;            // keys per tile
constexpr uint32_t kPollLimit = 1u << 22;  // look-back polls before giving up

template <int THREADS>
struct PassSmem {
  uint32_t keys[kPassTile];
  uint32_t vals[kPassTile];
  uint32_t warp_count[THREADS / 32][kRadix];
  uint32_t tile_offset[kRadix];   // exclusive scan of the tile's digit histogram
  int64_t global_base[kRadix];    // output index of staged slot 0 of each digit
  uint32_t scan_scratch[8];
  uint32_t tile_id;
  uint32_t abort;
};

// FIRST: the values are the particle indices themselves and are synthesised
// instead of read (the key kernel does not write an index array).
// Returns false when a look-back gave up.
template <bool FIRST, int THREADS>
__device__ __forceinline__ bool digit_pass(PassSmem<THREADS>& s, const uint32_t* keys_in,
                                           const uint32_t* vals_in, uint32_t* keys_out,
                                           uint32_t* vals_out, int64_t n, int shift,
                                           const uint32_t* digit_total, uint32_t* status,
                                           uint32_t* tile_counter, uint32_t tiles, int32_t* error,
                                           uint32_t poll_limit) {
  constexpr int kItems = kPassTile / THREADS;
  constexpr int kWarps = THREADS / 32;
  static_assert(kPassTile % THREADS == 0 && THREADS >= kRadix, "tile shape");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // A block works through tiles until none is left.  Tiles are handed out in
  // ticket order and a block holds one tile at a time, so every tile a block
  // waits on belongs to a block that is already running.
  if (tid == 0) s.abort = 0;
  for (;;) {
    if (tid == 0) s.tile_id = atomicAdd(tile_counter, 1u);
#pragma unroll
    for (int i = lane; i < kRadix; i += 32) s.warp_count[warp][i] = 0;
    __syncthreads();
    const uint32_t tile = s.tile_id;
    if (tile >= tiles) break;
    const int64_t tile_base = static_cast<int64_t>(tile) * kPassTile;
    const int valid = static_cast<int>(
        min(static_cast<long long>(kPassTile), static_cast<long long>(n - tile_base)));

    // Warp-striped load: item k of lane l is element warp*32*ITEMS + k*32 + l,
    // so (k, lane) order is index order.  Slots past the end get the largest key;
    // they rank after every real key of the last tile and are never written out.
    const int warp_first = warp * 32 * kItems + lane;
    uint32_t key[kItems], rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int e = warp_first + k * 32;
      key[k] = e < valid ? __ldcs(keys_in + tile_base + e) : 0xffffffffu;
    }

    // Stable rank inside the warp's segment: lanes with equal digits find each
    // other with match.any; the lowest of them advances the warp's counter.
    uint32_t* wc = s.warp_count[warp];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t d = (key[k] >> shift) & (kRadix - 1);
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const int leader = __ffs(peers) - 1;
      uint32_t before = 0;
      if (lane == leader) {
        before = wc[d];
        wc[d] = before + __popc(peers);
      }
      __syncwarp();
      rank[k] = __shfl_sync(0xffffffffu, before, leader) + __popc(peers & lanemask_lt());
    }
    __syncthreads();

    // Per digit: turn the warps' counts into exclusive offsets, publish the tile
    // aggregate, scan the tile histogram, look back.
    uint32_t tile_count = 0;
    if (tid < kRadix) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = s.warp_count[w][tid];
        s.warp_count[w][tid] = tile_count;
        tile_count += c;
      }
      st_relaxed(status + static_cast<size_t>(tile) * kRadix + tid,
                 tile_count | (tile == 0 ? kFlagInclusive : kFlagAggregate));
    }
    // Exclusive scans over the 256 digits (threads 0..255 = warps 0..7): the
    // tile's own histogram and the pass's global histogram.
    uint32_t total = 0, tile_excl = 0, total_excl = 0;
    if (tid < kRadix) {
      total = digit_total[tid];
      uint32_t a = tile_count, b = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t ta = __shfl_up_sync(0xffffffffu, a, o), tb = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) { a += ta; b += tb; }
      }
      if (lane == 31) {
        s.scan_scratch[warp] = a;
        s.tile_offset[warp] = b;  // borrowed as scratch until the barrier below
      }
      tile_excl = a - tile_count;
      total_excl = b - total;
    }
    __syncthreads();
    uint32_t tile_carry = 0, total_carry = 0;
    if (tid < kRadix) {
      for (int w = 0; w < warp; ++w) {
        tile_carry += s.scan_scratch[w];
        total_carry += s.tile_offset[w];
      }
    }
    __syncthreads();
    if (tid < kRadix) {
      tile_excl += tile_carry;
      total_excl += total_carry;
      s.tile_offset[tid] = tile_excl;
      // Decoupled look-back over the predecessors' status words of this digit.
      uint32_t exclusive = 0;
      bool gave_up = false;
      for (int64_t pred = static_cast<int64_t>(tile) - 1; pred >= 0; --pred) {
        const uint32_t* word_ptr = status + static_cast<size_t>(pred) * kRadix + tid;
        uint32_t word = ld_relaxed(word_ptr);
        uint32_t polls = 0;
        while ((word & kFlagMask) == 0) {
          if (++polls > poll_limit) { gave_up = true; break; }
          __nanosleep(32);
          word = ld_relaxed(word_ptr);
        }
        if (gave_up) break;
        exclusive += word & kValueMask;
        if ((word & kFlagMask) == kFlagInclusive) break;
      }
      if (gave_up) {
        atomicCAS(error, 0, kErrLookbackTimeout);
        s.abort = 1;
      }
      if (tile != 0)
        st_relaxed(status + static_cast<size_t>(tile) * kRadix + tid,
                   ((exclusive + tile_count) & kValueMask) | kFlagInclusive);
      s.global_base[tid] = static_cast<int64_t>(total_excl) + exclusive - tile_excl;
    }
    __syncthreads();

    // Stage the tile in digit order in shared memory.
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t d = (key[k] >> shift) & (kRadix - 1);
      rank[k] += s.tile_offset[d] + s.warp_count[warp][d];
      s.keys[rank[k]] = key[k];
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int e = warp_first + k * 32;
      uint32_t v;
      if (FIRST) v = static_cast<uint32_t>(tile_base + e);
      else v = e < valid ? __ldcs(vals_in + tile_base + e) : 0u;
      s.vals[rank[k]] = v;
    }
    __syncthreads();
    if (s.abort) return false;

    // Coalesced scatter: consecutive staged slots of one digit go to consecutive
    // output slots.
#pragma unroll 4
    for (int j = tid; j < valid; j += THREADS) {
      const uint32_t kk = s.keys[j];
      const int64_t dst = s.global_base[(kk >> shift) & (kRadix - 1)] + j;
      keys_out[dst] = kk;
      vals_out[dst] = s.vals[j];
    }
    __syncthreads();  // the staged tile and the ticket slot are reused by the next tile
  }
  return true;
}

// ------------------------------------------------------------------------
// cell_start from the sorted keys.
// ------------------------------------------------------------------------
// Position i in [0, n] is a boundary when its cell differs from the cell of
// position i-1 (cell -1 before the first key, cell C after the last).  The
// boundary thread writes `i` as the start of every cell in (previous, current];
// long runs of empty cells are filled by the whole warp.
template <int THREADS>
__device__ __forceinline__ void cell_bounds(const uint32_t* keys, int64_t n, int64_t num_cells,
                                            int32_t* cell_start, uint32_t block, uint32_t blocks) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = static_cast<int64_t>(blocks) * THREADS;
  const int64_t rounds = (n + 1 + stride - 1) / stride;
  for (int64_t r = 0; r < rounds; ++r) {
    const int64_t i = r * stride + static_cast<int64_t>(block) * THREADS + threadIdx.x;
    int64_t first = 0, last = -1;  // cells [first, last] start at i
    if (i <= n) {
      const int64_t cur = i < n ? static_cast<int64_t>(keys[i] >> kShuffleBits) : num_cells;
      const int64_t prev = i > 0 ? static_cast<int64_t>(keys[i - 1] >> kShuffleBits) : -1;
      first = prev + 1;
      last = cur;
    }
    const bool is_long = last - first >= 32;
    if (!is_long)
      for (int64_t c = first; c <= last; ++c) cell_start[c] = static_cast<int32_t>(i);
    uint32_t pending = __ballot_sync(0xffffffffu, is_long);
    while (pending) {
      const int src = __ffs(pending) - 1;
      pending &= pending - 1;
      const int64_t f = __shfl_sync(0xffffffffu, first, src);
      const int64_t l = __shfl_sync(0xffffffffu, last, src);
      const int32_t v = static_cast<int32_t>(__shfl_sync(0xffffffffu, i, src));
      for (int64_t c = f + lane; c <= l; c += 32) cell_start[c] = v;
    }
  }
}

// ------------------------------------------------------------------------
// Work in phases by the blocks of an ordinary launch.
// ------------------------------------------------------------------------
// A block may only wait for work that a running block has taken on: then it does not matter how
// many blocks of the launch run at the same time (a cooperative launch, which makes all of them
// resident, cannot start while another stream's kernel keeps one multiprocessor).
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

// Counts pieces of work as done, with all that the block has written.
__device__ __forceinline__ void arrive(uint32_t* done, uint32_t pieces = 1) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(done, pieces);
  }
}

// Waits until `*done & mask` reaches `target`; false, in every thread of the block, when that
// takes longer than `limit_ns` on the global timer or when some block has recorded an error.
// `last`: in thread 0, the whole word as it was then.
__device__ __forceinline__ bool wait_reaches(const uint32_t* done, uint32_t target,
                                             const int32_t* error, unsigned long long limit_ns,
                                             uint32_t mask = 0xffffffffu, uint32_t* last = nullptr) {
  bool stop = false;
  if (threadIdx.x == 0) {
    unsigned long long started = 0;
    for (;;) {
      uint32_t seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(done) : "memory");
      if (last) *last = seen;
      if ((seen & mask) >= target) break;
      if (ld_relaxed(reinterpret_cast<const uint32_t*>(error)) != 0) { stop = true; break; }
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (started == 0) started = now;
      else if (now - started > limit_ns) { stop = true; break; }
    }
    __threadfence();
  }
  return __syncthreads_or(stop) == 0;
}

// The same; a block that gives up records the error, and the others leave when they see it.
__device__ __forceinline__ bool wait_for(const uint32_t* done, uint32_t target, int32_t* error,
                                         unsigned long long limit_ns = kWaitLimitNs,
                                         uint32_t mask = 0xffffffffu, uint32_t* last = nullptr) {
  if (wait_reaches(done, target, error, limit_ns, mask, last)) return true;
  if (threadIdx.x == 0) atomicCAS(error, 0, kErrBarrierTimeout);
  return false;
}

// `phases` phases of `items` pieces of work each, whatever the number of blocks: piece k of the
// whole is item k % items of phase k / items.  Pieces are handed out in that order, and a block
// does one at a time, so all pieces of the phase it waits for belong to blocks that run.
// body(phase, item) returns false when the block must stop.
template <class Body>
__device__ __forceinline__ void run_phases(Header* hdr, uint32_t items, uint32_t phases, Body body) {
  __shared__ uint32_t turn;
  for (;;) {
    if (threadIdx.x == 0) turn = atomicAdd(&hdr->phase_ticket, 1u);
    __syncthreads();
    const uint32_t phase = turn / items, item = turn % items;
    if (phase >= phases) return;
    if (!wait_for(&hdr->phase_done, phase * items, &hdr->error)) return;
    if (!body(phase, item)) return;
    arrive(&hdr->phase_done);
  }
}

// ------------------------------------------------------------------------
// The whole digit-pass sort inside one launch.
// ------------------------------------------------------------------------
struct DigitPassArgs {
  const float *x, *y, *z, *v;
  int64_t padded, n, num_cells;
  AetherGrid grid;
  uint32_t k0, k1;
  PushSpec push;
  uint32_t* keys_out;
  int32_t* index_out;
  int32_t *cell_counts, *cell_start;
  float *xs, *ys, *zs, *vs;
  int64_t padded_sorted;
  // workspace of the digit passes
  int passes;
  uint32_t tiles;
  uint32_t* clear_from;   // words to zero before the first pass
  int64_t clear_words;
  uint32_t* status;
  uint32_t *keys_alt, *index_alt;
  float4* records;        // room for one 32-byte payload record per particle, or null
};

__device__ __forceinline__ uint32_t digit_phases(const DigitPassArgs& a) { return a.passes + 4; }

// Item `item` of `items` of phase `phase` of the sort; false when a look-back gave up.  The speed
// of this function matters little: it runs for calls whose density the bucketed path cannot hold.
template <int THREADS>
__device__ __forceinline__ bool digit_phase(const DigitPassArgs& a, PassSmem<THREADS>& s, Header* hdr,
                                            uint32_t phase, uint32_t item, uint32_t items) {
  const int64_t stride = static_cast<int64_t>(items) * THREADS;
  const int64_t first = static_cast<int64_t>(item) * THREADS + threadIdx.x;
  const bool odd = a.passes % 2 != 0;
  uint32_t* out_v = reinterpret_cast<uint32_t*>(a.index_out);
  uint32_t *cur_k = odd ? a.keys_alt : a.keys_out, *cur_v = odd ? a.index_alt : out_v;
  uint32_t *nxt_k = odd ? a.keys_out : a.keys_alt, *nxt_v = odd ? out_v : a.index_alt;

  if (phase == 0) {
    for (int64_t i = first; i < a.clear_words; i += stride) a.clear_from[i] = 0;
  } else if (phase == 1) {
    // Keys, digit histograms and payload records (with the move stage, if it is fused).
    uint32_t* hist = &s.warp_count[0][0];
    for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += THREADS) hist[i] = 0;
    __syncthreads();
    constexpr int kBatch = 2;  // particles whose loads are under way together
    const int64_t rounds = (a.n + kBatch * stride - 1) / (kBatch * stride);
    for (int64_t r = 0; r < rounds; ++r) {  // the same number for every thread: warp votes below
      float q[kBatch][6];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const int64_t i = (r * kBatch + k) * stride + first;
        const bool ok = i < a.n, moved = ok && a.records && a.v;
        q[k][0] = ok ? a.x[i] : 0.f;
        q[k][1] = ok ? a.y[i] : 0.f;
        q[k][2] = ok ? a.z[i] : 0.f;
        q[k][3] = moved ? a.v[i] : 0.f;
        q[k][4] = moved ? a.v[a.padded + i] : 0.f;
        q[k][5] = moved ? a.v[2 * a.padded + i] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const int64_t i = (r * kBatch + k) * stride + first;
        const bool ok = i < a.n;
        uint32_t key = 0;
        if (ok) {
          if (a.records) {
            if (a.push.enabled) {
#pragma unroll
              for (int c = 0; c < 3; ++c)
                push_axis(q[k][c], q[k][3 + c], a.push.dt, a.push.lo[c], a.push.hi[c]);
            }
            a.records[2 * i] = make_float4(q[k][0], q[k][1], q[k][2], q[k][3]);
            a.records[2 * i + 1] = make_float4(q[k][4], q[k][5], 0.f, 0.f);
          }
          key = make_key(cell_of(q[k][0], q[k][1], q[k][2], a.grid), static_cast<uint32_t>(i), a.k0, a.k1);
          cur_k[i] = key;
        }
        for (int p = 0; p < a.passes; ++p)
          bin_add(hist + p * kRadix, (key >> (kRadixBits * p)) & (kRadix - 1), ok);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.passes * kRadix; i += THREADS)
      if (hist[i]) atomicAdd(&hdr->digit_hist[0][0] + i, hist[i]);
  } else if (phase < static_cast<uint32_t>(a.passes) + 2) {
    const int p = static_cast<int>(phase) - 2;
    if (p % 2 != 0) {
      uint32_t* t = cur_k; cur_k = nxt_k; nxt_k = t;
      t = cur_v; cur_v = nxt_v; nxt_v = t;
    }
    uint32_t* st = a.status + static_cast<size_t>(p) * a.tiles * kRadix;
    return p == 0 ? digit_pass<true, THREADS>(s, cur_k, nullptr, nxt_k, nxt_v, a.n, 0,
                                              hdr->digit_hist[0], st, &hdr->tile_counter[0], a.tiles,
                                              &hdr->error, kPollLimit)
                  : digit_pass<false, THREADS>(s, cur_k, cur_v, nxt_k, nxt_v, a.n, kRadixBits * p,
                                               hdr->digit_hist[p], st, &hdr->tile_counter[p], a.tiles,
                                               &hdr->error, kPollLimit);
  } else if (phase == static_cast<uint32_t>(a.passes) + 2) {
    if (a.xs) {
      constexpr int kBatch = 4;  // particles whose loads are under way together
      for (int64_t r0 = first; r0 < a.n; r0 += kBatch * stride) {
        float4 lo[kBatch], hi[kBatch];
        int32_t index[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          const int64_t r = r0 + k * stride;
          index[k] = r < a.n ? __ldcg(a.index_out + r) : 0;
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          const int64_t i = index[k];
          if (a.records) {
            lo[k] = __ldcg(a.records + 2 * i);
            hi[k] = __ldcg(a.records + 2 * i + 1);
          } else {
            lo[k] = make_float4(a.x[i], a.y[i], a.z[i], a.v ? a.v[i] : 0.f);
            hi[k] = make_float4(a.v ? a.v[a.padded + i] : 0.f, a.v ? a.v[2 * a.padded + i] : 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          const int64_t r = r0 + k * stride;
          if (r >= a.n) break;
          a.xs[r] = lo[k].x;
          a.ys[r] = lo[k].y;
          a.zs[r] = lo[k].z;
          if (a.vs) {
            a.vs[r] = lo[k].w;
            a.vs[a.padded_sorted + r] = hi[k].x;
            a.vs[2 * a.padded_sorted + r] = hi[k].y;
          }
        }
      }
    }
    cell_bounds<THREADS>(a.keys_out, a.n, a.num_cells, a.cell_start, item, items);
  } else {
    for (int64_t c = first; c < a.num_cells; c += stride)
      a.cell_counts[c] = __ldcg(a.cell_start + c + 1) - __ldcg(a.cell_start + c);
  }
  return true;
}

}  // namespace aether
