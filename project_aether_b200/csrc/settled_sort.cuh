// The sort of a moved state that starts cell-sorted (included by sort_bucketed.cu).
//
// A time-stepping loop sorts the particles, moves them a little, and sorts them again: the input is
// in the order of the cells its particles were in, and most of them are still there.  The buckets
// of the general path take every particle through a record in HBM; here only those that left their
// bucket (movers) travel so, and the others are read from the input where they lie:
//
//   settled_probe_kernel   clears the tables, and looks at a sample of the particles: how many leave their
//                          bucket, and whether they are in bucket order
//   settled_scan_kernel    reads the input once and moves the particles: their keys; where every
//                          bucket's particles lie in the input (its home run; the input must be in
//                          bucket order, before the move); who leaves which bucket, and the movers'
//                          records into lists, one per block
//   settled_sums_kernel,   where every bucket's arrivals and its output begin; groups of buckets
//   settled_groups_kernel
//   settled_movers_kernel  the lists' records to their buckets' arrivals
//   settled_finish_kernel  a block takes a group: reads its home run and keys, moves the particles once
//                          more, leaves out those that left, adds the arrivals, sorts and writes the group
//   bucket_finish_kernel   (of the general path) the same for dense regions, whose buckets those blocks do not hold
//   bucket_tail_kernel     the same for single buckets that the kernel before does not hold
//
// It moves 24 + 4 + 28 + 32 bytes per particle, and some 130 more per mover, where the general path moves
// 24 + 24 + 32 + 32 + 32.  Bound by instructions: with the keys made in the finish kernel, 24 + 24 + 32
// bytes, 128 M particles took 3499 us (scan 684, finish 2649) where with keys from the scan they took 3248 (897, 2071;
// the finish now 1560).
//
// Whether the input is in order, and how many particles move, is only known on the device.  Whatever
// speaks against the path sets Header::settle_failed; the kernels above then stop, and the general path's
// kernels, which are enqueued behind them and otherwise return at once, do the call from the start.  When
// it is noticed: random order and too many movers by the probe; a particle out of order, or more movers than
// the lists hold in one part of the input, in the round of the scan that meets it; a counter that wraps in
// the finish.  Buckets of a dense region are no reason.  Calls that the probe gives up, without the attempt / with
// it, particles that have all left their cell: 1.6 M 74 / 91 us, 4 M 162 / 176, 6 M 225 / 240, 16.8 M 551 / 567, 30 M 909 / 925, 64 M
// 1951 / 1965, 128 M 3848 / 3890; in random order 1.6 M 77 / 91, 4 M 164 / 176, 16.8 M 599 / 614, 64 M 2239 / 2252.

constexpr int kSettledThreads = 512;
constexpr int kSettledRound = kSettledThreads * 4;  // particles of a block per round
constexpr int kListShare = 2;                       // a block's list has room for one mover in two particles
constexpr int kMoverShare = 4;                      // all lists together for one in four
constexpr int kProbeSamples = 128;                  // particles of each of the scan's blocks that the probe looks at
constexpr int kSettledPart = 4096;                  // buckets per entry of the coarse sums
constexpr int kSettledSums = 4 * (1 + kSettledPart / kGroupSpan);  // words of such an entry: of the part, of its kGroupSpan buckets each
constexpr int kDenseSpanLog = 3;                    // buckets that are dense or not together
constexpr int kSettledWideShare = 1024;             // particles to a bucket above a dense group's capacity, at least
constexpr uint32_t kGone = 0xffffffffu;             // no key: grids of 2^25 cells are left to the general path
constexpr int kSettledRowWords = 8;                 // words of a group's table
// What sorts a group in the finish: THREADS threads that hold ITEMS records each, move and all, in registers.
template <int THREADS, int ITEMS, int LOW_BITS>
struct SettledShape {
  static constexpr int kThreads = THREADS, kItems = ITEMS, kLowBits = LOW_BITS;
  static constexpr int kBlocks = 1024 / THREADS;          // per multiprocessor, 64 registers a thread
  static constexpr int kCapacity = THREADS * ITEMS;
  static constexpr int kHistWords = (1 << LOW_BITS) / 4;  // byte counters, four to a word
  static constexpr int kWordsPerThread = kHistWords / THREADS;
  static constexpr int kMaxDrop = 2, kMostIndexBits = 0;  // see FinishShape
  static constexpr int kMaxCells = 1 << (LOW_BITS + kMaxDrop - kShuffleBits);
  static_assert(kWordsPerThread % 4 == 0 && THREADS <= 1024, "the counter scan reads four words at a time");
};
// Teams are the usual shape: a group's barriers hold up four warps only, and eight groups share a
// multiprocessor (finish of 16.8 M particles, 8 to a cell: 199 us; 256 threads that hold 1024 records 213, 512 that
// hold 2048 242, 64 that hold 256 214; three items a thread 217, six 220, eight 279, which leave fewer threads).  Their
// groups span 64 cells at most, so that sparse grids do not fill them, and a cell may have some 400 particles: beyond
// either limit the groups are blocks' (20 M particles, 4 / 5 / 6 to a cell: teams 351 / 300 / 253 us, blocks 285 /
// 286 / 286).  Where the density differs from place to place, spans of 2^kDenseSpanLog buckets with one above a
// team's capacity are cut into groups of SettledDense, which the general path's finish kernel sorts, otherwise idle then; a
// bucket that those do not hold is a whole block's of the tail kernel, SettledWide, up to its capacity.
// us per call before teams / with all 256 buckets around such a bucket in groups of 4096 places, one to a multiprocessor, in the tail
// kernel / this, share of the particles in a share of the space: 4 M in 79^3 cells, 0.1 in 0.01 142 / 159 / 134, 0.28 in 0.03
// 162 / 157 / 141; 16.8 M in 112^3, 0.5 in 0.05 476 / 543 / 477, 0.5 in 0.1 466 / 525 / 453; 64 M in 175^3 1638 / 1804 / 1644, 1609 / 1752 / 1550.
// Worst where a bucket is just above half of a dense group: 2.5 M in 59^3, 0.5 in 0.05 105 / 133 / 115; 30 M in 67^3
// 868 / 966 / 918.  (Dense groups of 2560 places, five records a thread: 110, 874, but 5 to 7 percent more elsewhere.  Two parts of a block of the
// tail kernel instead of the finish kernel: 130, 1060.  Buckets half as wide: 2 percent more where the density is even.)
using SettledTeam = SettledShape<128, 4, 11>;
using SettledBlock = SettledShape<512, 4, 14>;
// Below some four fifths of a particle to a cell a group is short of records, not of cells, and what it costs is its 2^14
// counters and the places that stay empty: few records a thread, four groups to a multiprocessor.  us per call before groups were
// sorted from registers / by SettledBlock / by this: 1.6 M in 160^3 cells 155 / 165 / 117, in 140^3 124 / 128 / 98, 17 M
// in 320^3 1068 / 1115 / 758, in 290^3 880 / 891 / 627 (512 threads with one record each 126, 102, 817, 678; with two 141, 111,
// 923, 749; 256 with four 130, 107, 855, 699; 128 with four 168, 138, 1173, 953).
using SettledSparse = SettledShape<256, 2, 14>;
using SettledDense = SettledBlock;
using SettledWide = SettledShape<1024, 4, 15>;
constexpr int64_t kSettledSparseMost = 400;    // particles on its most cells, on average at most: of 512 places
constexpr int64_t kSettledTeamLeast = 352;     // particles on a team's most cells, on average at least
constexpr int64_t kSettledTeamMostMean = 384;  // particles of a cell, on average at most
// Records per bucket, on average at most.  Buckets cost this path little (a few words each), and with
// five or more to a group the groups fill a team, or a block (teams, 16.8 M particles: 64 to a bucket 443 us per
// call, 128 450).
constexpr int64_t kSettledTeamTarget = 104, kSettledBlockTarget = 320;
// Where single cells hold more than this on average, the buckets of the path would not fit a block.
constexpr int64_t kSettledMostMean = 1024;

struct SettledArgs {
  const float *x, *y, *z, *v;
  int64_t padded, num_cells;
  int n;
  PushSpec push;
  AetherGrid grid;
  uint32_t k0, k1;
  int shift, buckets;
  int per_block;          // particles per block of the scan, a multiple of kSettledRound
  int scan_blocks;
  uint32_t capacity;      // of the shape that sorts the usual groups
  int most_cells;
  uint32_t most_sampled;  // movers of the sample from which on the general path is faster
  uint32_t most_movers;   // what fits `arrived`
  uint32_t *first, *end;            // [buckets] home run in the input; both zero if it is empty
  uint32_t *leavers, *arrivals;     // [buckets]
  uint32_t* keys;                   // [n] key of every particle after the move, kGone of those that left
  uint32_t* list_count;             // [scan_blocks] movers found by each block of the scan
  uint32_t* cursor;                 // [buckets] next free place of each bucket's arrivals
  uint32_t* sums;                   // [parts][kSettledSums] particles at home, arrivals, output of kSettledPart buckets
  uint32_t* tables;                 // [buckets][kSettledRowWords]: groups of teams, and from the end buckets in no group
  uint32_t* dense_tables;           // [buckets][kSettledRowWords]: groups of dense regions
  uint32_t* wide_tables;            // [n / kSettledWideShare + 1][kSettledRowWords]: buckets that those do not hold
  uint32_t *list, *arrived;         // records: the movers block by block, and bucket by bucket
  int vec_out;            // the outputs take 16-byte stores where the place is a multiple of four
  Header* hdr;
};

__device__ __forceinline__ bool settle_failed(const Header* hdr) {
  return ld_relaxed(&hdr->settle_failed) != 0;
}
__device__ __forceinline__ void fail_settle(Header* hdr) { atomicExch(&hdr->settle_failed, 1u); }

// The move and the cell of a particle with little arithmetic: walls are looked at together, and
// the reflection is done by the few that hit one.  WHOLE: the slab is the whole grid.
__device__ __forceinline__ void push_particle(const PushSpec& push, float* f) {
  bool hit = false;
  float moved[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    moved[c] = __fadd_rn(f[c], __fmul_rn(f[3 + c], push.dt));
    hit |= moved[c] < push.lo[c] || moved[c] > push.hi[c];
  }
  if (hit) {
#pragma unroll
    for (int c = 0; c < 3; ++c) push_axis(f[c], f[3 + c], push.dt, push.lo[c], push.hi[c]);
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] = moved[c];
  }
}
template <bool WHOLE>
__device__ __forceinline__ uint32_t settled_cell(float x, float y, float z, const AetherGrid& g) {
  if (!WHOLE) return cell_of(x, y, z, g);
  const int ix = axis_index(x, g.x0, g.inv_dx, g.nx);
  const int iy = axis_index(y, g.y0, g.inv_dy, g.ny);
  const int iz = axis_index(z, g.z0, g.inv_dz, g.nz);
  return static_cast<uint32_t>((iz * g.ny + iy) * g.nx + ix);
}

// What a warp of the scan keeps in shared memory: the movers it has found and not yet stored.  A
// round adds at most 128 to fewer than 32.
struct MoverQueue {
  uint4 record[160][2];  // {cell, index, x, y}, {z, vx, vy, vz}
};

// Stores 32 (or, at the end, the last `count`) of a warp's movers in the block's list; false if
// there is no room.
__device__ __forceinline__ bool flush_movers(const SettledArgs& a, const MoverQueue& queue, int from, int count,
                                             uint32_t* fill, uint32_t room, uint32_t* list) {
  const int lane = lane_id();
  uint32_t place = 0;
  if (lane == 0) place = atomicAdd(fill, static_cast<uint32_t>(count));
  place = __shfl_sync(0xffffffffu, place, 0);
  if (place + count > room) return false;
  if (lane < count) {
    const uint4 lo = queue.record[from + lane][0], hi = queue.record[from + lane][1];
    atomicAdd(&a.arrivals[lo.x >> a.shift], 1u);
    store_record(list + static_cast<size_t>(place + lane) * kRecordWords, lo.x, lo.y, __uint_as_float(lo.z),
                 __uint_as_float(lo.w), __uint_as_float(hi.x), __uint_as_float(hi.y), __uint_as_float(hi.z),
                 __uint_as_float(hi.w));
  }
  __syncwarp();  // the queue is written again
  return true;
}

// One round of a block: four particles per thread, from i0 = this thread's first.  FULL: none of the
// block's round is missing.  Returns what a lane found against the input's order.
template <bool VEC, bool WHOLE, bool FULL>
__device__ __forceinline__ bool scan_round(const SettledArgs& a, int i0, int last, MoverQueue& queue, int& queued) {
  const int lane = lane_id();
  float f[6][4];
  if (FULL && VEC) {
    load_items<4>(a.x + i0, f[0]);
    load_items<4>(a.y + i0, f[1]);
    load_items<4>(a.z + i0, f[2]);
    load_items<4>(a.v + i0, f[3]);
    load_items<4>(a.v + a.padded + i0, f[4]);
    load_items<4>(a.v + 2 * a.padded + i0, f[5]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool ok = FULL || last - i0 > k;
      f[0][k] = ok ? a.x[i0 + k] : 0.f;
      f[1][k] = ok ? a.y[i0 + k] : 0.f;
      f[2][k] = ok ? a.z[i0 + k] : 0.f;
      f[3][k] = ok ? a.v[i0 + k] : 0.f;
      f[4][k] = ok ? a.v[a.padded + i0 + k] : 0.f;
      f[5][k] = ok ? a.v[2 * a.padded + i0 + k] : 0.f;
    }
  }
  // The bucket of the particle before a warp's first one.
  uint32_t before = 0;
  if (lane == 0 && i0 > 0 && (FULL || i0 < last))
    before = settled_cell<WHOLE>(a.x[i0 - 1], a.y[i0 - 1], a.z[i0 - 1], a.grid) >> a.shift;
  uint32_t home[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) home[k] = settled_cell<WHOLE>(f[0][k], f[1][k], f[2][k], a.grid) >> a.shift;
  const uint32_t left = __shfl_up_sync(0xffffffffu, home[3], 1);
  if (lane > 0) before = left;
  bool bad = false;
  uint32_t found[4], key[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool valid = FULL || last - i0 > k;
    if (valid && home[k] != before && i0 + k > 0) {
      bad |= home[k] < before;
      a.first[home[k]] = static_cast<uint32_t>(i0 + k);
      a.end[before] = static_cast<uint32_t>(i0 + k);
    }
    before = home[k];
    float q[6] = {f[0][k], f[1][k], f[2][k], f[3][k], f[4][k], f[5][k]};
    push_particle(a.push, q);
    const uint32_t cell = settled_cell<WHOLE>(q[0], q[1], q[2], a.grid);
    const bool moved = valid && cell >> a.shift != home[k];
    found[k] = __ballot_sync(0xffffffffu, moved);
    key[k] = moved ? kGone : make_key(cell, static_cast<uint32_t>(i0 + k), a.k0, a.k1);
    if (moved) {
      atomicAdd(&a.leavers[home[k]], 1u);
      uint4* to = queue.record[queued + __popc(found[k] & lanemask_lt())];
      to[0] = make_uint4(cell, static_cast<uint32_t>(i0 + k), __float_as_uint(q[0]), __float_as_uint(q[1]));
      to[1] = make_uint4(__float_as_uint(q[2]), __float_as_uint(q[3]), __float_as_uint(q[4]), __float_as_uint(q[5]));
    }
    queued += __popc(found[k]);
  }
  if (FULL) {
    *reinterpret_cast<uint4*>(a.keys + i0) = make_uint4(key[0], key[1], key[2], key[3]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (last - i0 > k) a.keys[i0 + k] = key[k];
  }
  return bad;
}

// Clears the tables of the scan and takes a sample of its particles, evenly spaced, with each one's neighbour.
// Bound by the latency of one access to HBM, which is hidden beside the kernel that zeroes the header: the inputs
// are read before the wait.  In place of a clear of the tables alone, which took a launch too: 4 M particles
// 143.5 -> 144.5 us per call, 1.6 M 81.5 -> 79.3, 16.8 M alike.
template <bool WHOLE>
__global__ void __launch_bounds__(kSettledThreads)
settled_probe_kernel(const __grid_constant__ SettledArgs a, int64_t pieces) {
  chain_release();
  const int tid = threadIdx.x;
  const int i = blockIdx.x * a.per_block + tid * (a.per_block / kProbeSamples);
  const bool sampled = tid < kProbeSamples && i < a.n;
  float f[6] = {}, next[3] = {};
  const int j = min(i + 1, a.n - 1);
  if (sampled) {
    f[0] = a.x[i];
    f[1] = a.y[i];
    f[2] = a.z[i];
    f[3] = a.v[i];
    f[4] = a.v[a.padded + i];
    f[5] = a.v[2 * a.padded + i];
    next[0] = a.x[j];
    next[1] = a.y[j];
    next[2] = a.z[j];
  }
  uint4* tables = reinterpret_cast<uint4*>(a.first);
  for (int64_t p = blockIdx.x * static_cast<int64_t>(kSettledThreads) + tid; p < pieces; p += gridDim.x * kSettledThreads)
    tables[p] = make_uint4(0u, 0u, 0u, 0u);
  const uint32_t home = settled_cell<WHOLE>(f[0], f[1], f[2], a.grid) >> a.shift;
  const bool unordered = sampled && settled_cell<WHOLE>(next[0], next[1], next[2], a.grid) >> a.shift < home;
  push_particle(a.push, f);
  const bool moved = sampled && settled_cell<WHOLE>(f[0], f[1], f[2], a.grid) >> a.shift != home;
  chain_wait();  // the header is zero; inputs and tables were free before the kernel that zeroes it began
  const int movers = __syncthreads_count(moved);
  const bool fail = __syncthreads_or(unordered) || movers > kProbeSamples / kListShare;  // more than the block's list holds
  if (tid == 0) {
    if (movers) atomicAdd(&a.hdr->settle_sampled, static_cast<uint32_t>(movers));
    if (fail) fail_settle(a.hdr);
  }
}

// Bound by instructions (65 % of the issue slots; HBM would take half the time).  The home runs are
// written where a bucket begins and where the bucket before it ends.  A mover costs two adds and a record
// of {cell, index, moved state}, which goes through the warp's queue so that 32 of them are
// stored at a time: stored one by one, under a branch per particle, 128 M took 761 us without keys, now 684.
template <bool VEC, bool WHOLE>
__global__ void __launch_bounds__(kSettledThreads, 2)
settled_scan_kernel(const __grid_constant__ SettledArgs a) {
  // No early release: the waiting blocks of the kernels behind would stand beside these (4 M particles 144.5 ->
  // 141.9 us per call, 16.8 M 467 -> 461, 64 M 1593 -> 1583).
  chain_wait();
  __shared__ uint32_t fill, stop;
  extern __shared__ MoverQueue queues[];
  const int tid = threadIdx.x, lane = tid & 31;
  MoverQueue& queue = queues[tid >> 5];
  // One answer for the block: others may set the word meanwhile.
  const bool refused = a.hdr->settle_sampled > a.most_sampled;
  if (tid == 0) {
    fill = stop = 0;
    if (refused && blockIdx.x == 0) fail_settle(a.hdr);
  }
  if (__syncthreads_or(refused || (tid == 0 && settle_failed(a.hdr)))) return;
  const int block_first = blockIdx.x * a.per_block;
  const int last = min(a.n - block_first, a.per_block) + block_first;
  const uint32_t room = static_cast<uint32_t>(a.per_block / kListShare);
  uint32_t* list = a.list + static_cast<size_t>(blockIdx.x) * room * kRecordWords;
  // The two ends of the input; the places between are the rounds' business.
  if (tid == 0 && blockIdx.x == 0) a.first[settled_cell<WHOLE>(a.x[0], a.y[0], a.z[0], a.grid) >> a.shift] = 0;
  if (tid == 0 && last == a.n)
    a.end[settled_cell<WHOLE>(a.x[last - 1], a.y[last - 1], a.z[last - 1], a.grid) >> a.shift] = static_cast<uint32_t>(a.n);
  int queued = 0;
  bool going = true;
  for (int i = block_first, r = 0; going && i < last; i += kSettledRound, ++r) {
    const int i0 = i + tid * 4;
    const bool seen = last - i >= kSettledRound ? scan_round<VEC, WHOLE, true>(a, i0, last, queue, queued)
                                                : scan_round<VEC, WHOLE, false>(a, i0, last, queue, queued);
    bool bad = __any_sync(0xffffffffu, seen);  // one answer for the warp, as all below
    __syncwarp();
    while (queued >= 32 && !bad) {
      queued -= 32;
      bad = !flush_movers(a, queue, queued, 32, &fill, room, list);
    }
    if (bad) {
      if (lane == 0) {
        *static_cast<volatile uint32_t*>(&stop) = 1;
        fail_settle(a.hdr);
      }
      going = false;
    } else {
      if (tid == 0 && r % 4 == 3 && settle_failed(a.hdr)) *static_cast<volatile uint32_t*>(&stop) = 1;
      going = !__any_sync(0xffffffffu, *static_cast<volatile uint32_t*>(&stop));
    }
  }
  if (going && queued > 0 && !flush_movers(a, queue, 0, queued, &fill, room, list) && lane == 0) fail_settle(a.hdr);
  __syncthreads();
  if (tid == 0) a.list_count[blockIdx.x] = min(fill, room);
}

// Particles at home before the move, arrivals and output of every kSettledPart buckets, and of every kGroupSpan.
__global__ void __launch_bounds__(1024)
settled_sums_kernel(const __grid_constant__ SettledArgs a) {
  chain_begin();
  if (settle_failed(a.hdr)) return;
  __shared__ uint32_t sum[kSettledSums];
  for (int i = threadIdx.x; i < kSettledSums; i += 1024) sum[i] = 0;
  __syncthreads();
  const int b0 = blockIdx.x * kSettledPart;
#pragma unroll
  for (int k = 0; k < kSettledPart / 1024; ++k) {
    const int at = k * 1024 + threadIdx.x, b = b0 + at;
    uint32_t home = 0, arrivals = 0, left = 0;
    if (b < a.buckets) {
      home = a.end[b] - a.first[b];
      arrivals = a.arrivals[b];
      left = a.leavers[b];
    }
    home = __reduce_add_sync(0xffffffffu, home);
    arrivals = __reduce_add_sync(0xffffffffu, arrivals);
    left = __reduce_add_sync(0xffffffffu, left);
    if ((threadIdx.x & 31) < 2) {  // lane 0 adds to the part's sums, lane 1 to its kGroupSpan buckets'
      uint32_t* to = sum + ((threadIdx.x & 31) == 0 ? 0 : 4 * (1 + at / kGroupSpan));
      atomicAdd(to, home);
      atomicAdd(to + 1, arrivals);
      atomicAdd(to + 2, home + arrivals - left);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kSettledSums; i += 1024) a.sums[blockIdx.x * kSettledSums + i] = sum[i];
}

// A block takes kGroupSpan consecutive buckets; it adds up what lies before them for itself, from the sums.
// Groups as in group_kernel; a bucket needs a place for each of its particles at home and each of its arrivals.
// A group's table: first particle of its home run, particles in it, first of its arrivals, arrivals, first
// output slot, records, its buckets b0, b1.  Runs of spans with a bucket that is more than a team holds have lists of their own,
// of dense groups and of single buckets that no such group holds; a bucket that no block holds gets a table from the end of
// the first array (there are no more groups and such buckets than buckets).  aux_counter[2], [3], [5], [4]: the four kinds.
__global__ void __launch_bounds__(kGroupSpan)
settled_groups_kernel(const __grid_constant__ SettledArgs a) {
  chain_begin();
  // One answer for the block: others may set the word meanwhile.
  if (__syncthreads_or(threadIdx.x == 0 && settle_failed(a.hdr))) return;
  __shared__ GroupCut cut;
  __shared__ uint32_t base[3];  // at home, arrivals, output before the block's buckets
  __shared__ uint32_t arrived[kGroupSpan + 1], output[kGroupSpan + 1];
  const int tid = threadIdx.x;
  const int b0 = blockIdx.x * kGroupSpan;
  const int here = min(kGroupSpan, a.buckets - b0);
  if (tid < 3) base[tid] = 0;
  __syncthreads();
  uint32_t before[3] = {0, 0, 0};
  const int part = b0 / kSettledPart, spans = (b0 - part * kSettledPart) / kGroupSpan;
  for (int p = tid; p < part + spans; p += kGroupSpan) {
    const uint32_t* sums = a.sums + (p < part ? p * kSettledSums : part * kSettledSums + 4 * (1 + p - part));
#pragma unroll
    for (int c = 0; c < 3; ++c) before[c] += sums[c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint32_t sum = __reduce_add_sync(0xffffffffu, before[c]);
    if ((tid & 31) == 0 && sum) atomicAdd(&base[c], sum);
  }
  uint32_t home = 0, in = 0, left = 0;
  if (tid < here) {
    home = a.end[b0 + tid] - a.first[b0 + tid];
    in = a.arrivals[b0 + tid];
    left = a.leavers[b0 + tid];
  }
  // Places (home + arrivals), arrivals and output before each bucket.
  const uint32_t places = block_exclusive_scan(home + in, cut.warp_sum, &cut.found);
  cut.start[tid] = places;
  if (tid == here - 1) cut.start[here] = cut.found;
  __syncthreads();
  const uint32_t arrivals = block_exclusive_scan(in, cut.warp_sum, &cut.found);
  arrived[tid] = arrivals;
  if (tid == here - 1) arrived[here] = cut.found;
  __syncthreads();
  const uint32_t written = block_exclusive_scan(home + in - left, cut.warp_sum, &cut.found);
  output[tid] = written;
  if (tid == here - 1) output[here] = cut.found;
  if (tid < here) a.cursor[b0 + tid] = base[1] + arrivals;
  __syncthreads();
  if (tid == 0 && base[1] + arrived[here] > a.most_movers) fail_settle(a.hdr);  // more than there is room for
  const uint32_t mine = tid < here ? cut.start[tid + 1] - cut.start[tid] : 0u;
  const int crowded = __syncthreads_count(mine > a.capacity);
  if (crowded && tid == 0) atomicAdd(&a.hdr->settle_large, static_cast<uint32_t>(crowded));
  // Dense spans, a bit each: a run of such, or of others, is cut into groups by itself.
  __shared__ uint32_t dense_spans;
  if (tid == 0) dense_spans = 0;
  __syncthreads();
  if (crowded && a.capacity < SettledDense::kCapacity && mine > a.capacity) atomicOr(&dense_spans, 1u << (tid >> kDenseSpanLog));
  __syncthreads();
  const int span = tid >> kDenseSpanLog;
  const bool dense = (dense_spans >> span) & 1u;
  const uint32_t unlike = dense ? ~dense_spans : dense_spans;
  const bool begins = tid == 0 || ((tid & ((1 << kDenseSpanLog) - 1)) == 0 && ((unlike >> (span - 1)) & 1u));
  const int next = __ffs(static_cast<int>(unlike & ~((2u << span) - 1)));  // one more than the next unlike span, or 0
  const uint32_t capacity = dense ? SettledDense::kCapacity : a.capacity;
  cut_groups_of_block(cut, here, begins, next ? (next - 1) << kDenseSpanLog : kGroupSpan, kGroupSpan,
                      (dense ? SettledDense::kMaxCells : a.most_cells) >> a.shift, capacity, &a.hdr->aux_counter[2],
                      &a.hdr->aux_counter[3], dense);
  auto write_table = [&](uint32_t* tables, uint32_t row, int first, int end) {
    uint4* table = reinterpret_cast<uint4*>(tables + static_cast<size_t>(row) * kSettledRowWords);
    const uint32_t in_group = arrived[end] - arrived[first];
    table[0] = make_uint4(base[0] + cut.start[first] - arrived[first],
                          cut.start[end] - cut.start[first] - in_group, base[1] + arrived[first], in_group);
    table[1] = make_uint4(base[2] + output[first], output[end] - output[first],
                          static_cast<uint32_t>(b0 + first), static_cast<uint32_t>(b0 + end));
  };
  const int found = static_cast<int>(cut.found), all = found + static_cast<int>(cut.found_other);
  if (tid < all)
    write_table(tid < found ? a.tables : a.dense_tables, tid < found ? cut.list_base + tid : cut.other_base + tid - found,
                cut.group_first[tid], cut.link[cut.group_first[tid]]);
  if (mine > SettledWide::kCapacity) write_table(a.tables, a.buckets - 1 - atomicAdd(&a.hdr->aux_counter[4], 1u), tid, tid + 1);
  else if (mine > capacity) write_table(a.wide_tables, atomicAdd(&a.hdr->aux_counter[5], 1u), tid, tid + 1);
}

// The movers' records to their buckets, with their keys.
__global__ void __launch_bounds__(kSettledThreads)
settled_movers_kernel(const __grid_constant__ SettledArgs a) {
  // No early release, so that the finish is placed on free multiprocessors (chained to this and let in at once /
  // at its end: 16.8 M particles 464 / 460 us per call, 64 M 1592 / 1580; an ordinary launch 463 / 1582, 2.6 M 106.2
  // against 103.8).
  chain_wait();
  if (settle_failed(a.hdr)) return;
  const uint32_t room = static_cast<uint32_t>(a.per_block / kListShare);
  const uint4* list = reinterpret_cast<const uint4*>(a.list + static_cast<size_t>(blockIdx.x) * room * kRecordWords);
  const uint32_t count = a.list_count[blockIdx.x];
#pragma unroll 2
  for (uint32_t j = threadIdx.x; j < count; j += kSettledThreads) {
    const uint4 lo = __ldcs(list + 2 * j), hi = __ldcs(list + 2 * j + 1);
    const uint32_t slot = atomicAdd(&a.cursor[lo.x >> a.shift], 1u);
    store_record(a.arrived + static_cast<size_t>(slot) * kRecordWords, make_key(lo.x, lo.y, a.k0, a.k1), lo.y,
                 __uint_as_float(lo.z), __uint_as_float(lo.w), __uint_as_float(hi.x), __uint_as_float(hi.y),
                 __uint_as_float(hi.z), __uint_as_float(hi.w));
  }
}

// Asks for the whole 16-byte pieces of [from, from + bytes) in L2.
__device__ __forceinline__ void prefetch_range(const void* from, uint32_t bytes) {
  const uintptr_t p0 = (reinterpret_cast<uintptr_t>(from) + 15) & ~uintptr_t{15};
  const uintptr_t p1 = (reinterpret_cast<uintptr_t>(from) + bytes) & ~uintptr_t{15};
  if (p1 > p0)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p0), "r"(static_cast<uint32_t>(p1 - p0)) : "memory");
}

template <class Shape>
struct __align__(16) SettledSmem {
  static constexpr int kRow = Shape::kCapacity + 4;
  uint32_t hist[Shape::kHistWords];
  union {
    struct {
      uint32_t tie[Shape::kCapacity + 4];  // the last words are read, but not used, behind the last run
      uint16_t word_prefix[Shape::kHistWords];
    };
    uint32_t stage[kRecordWords][kRow];  // the output, array by array
  };
  uint32_t warp_sum[32];
};

// What the kernels behind the sort of a settled state know of it.
struct SettledCall {
  SettledArgs args;
  FinishOut out;
};

struct BlockBarrier {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
// Of the THREADS threads of a part of a block.
template <int THREADS>
struct PartBarrier {
  int part;
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync %0, %1;" ::"r"(part + 1), "n"(THREADS) : "memory");
  }
};

// Groups g, g + step, ... of a list, one after the other; false if a counter wrapped.  The sort is that of
// sort_placed: byte counters of the low key, whose returned value is the rank on a counter, their scan, and a compare
// of the records that share one.  But a thread keeps its records in registers from load to store, and puts them in
// output order in shared memory array by array, so that the output goes out 16 bytes at a time: a record costs eight
// stores of a word at one address with constant offsets and a quarter of eight loads and stores of 16 bytes, where
// whole records, pulled out of shared memory by sorted place, cost four accesses of 16 bytes, eight stores of a word and
// their addresses.  The bodies of the item loops are written so that the compiler predicates single accesses
// instead of branching around them (325 -> 229 instructions a record).  Bound by instructions and the
// shared-memory pipe (issue slots 54 %, pipe 74 %).  16.8 M particles, 8 to a cell, 285 -> 199 us, 20 M with 64
// 344 -> 253, 128 M 2168 -> 1560 (60 bytes a particle: 5.2 TB/s).  Stored to the output straight from the
// registers, neighbouring lanes to places a few cells wide, 16.8 M took 221 us in groups of 1024, and 64 to a cell
// 372, in parts of sectors; read by sorted place instead, 250 and 299.
template <class Shape, class Barrier>
__device__ __forceinline__ bool finish_settled_groups(SettledSmem<Shape>& s, const SettledArgs& a, const FinishOut& out,
                                                      const uint32_t* list, uint32_t g, uint32_t groups, uint32_t step,
                                                      int tid, Barrier barrier) {
  constexpr int kThreads = Shape::kThreads, kItems = Shape::kItems, kWarps = kThreads / 32;
  constexpr int kWordsPerThread = Shape::kWordsPerThread;
  const int lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < Shape::kHistWords; i += kThreads) s.hist[i] = 0;
  const uint4* tables = reinterpret_cast<const uint4*>(list);  // two to a group
  uint4 where{}, what{};
  if (g < groups) {
    where = tables[2 * g];
    what = tables[2 * g + 1];
  }
  for (; g < groups; g += step) {
    const uint32_t home_first = where.x, home = where.y, places = home + where.w, first_arrived = where.z;
    const uint32_t begin = what.x, count = what.y;
    const uint32_t first_cell = what.z << a.shift;
    const int cells_here = min(static_cast<int>((what.w << a.shift) - first_cell),
                               static_cast<int>(a.num_cells - first_cell));
    float f[kItems][6];
    uint32_t key[kItems], word[kItems];
    {
      const uint32_t mine = home_first + tid;
      const uint32_t* keys = a.keys + mine;
      const float *x = a.x + mine, *y = a.y + mine, *z = a.z + mine;
      const float *vx = a.v + mine, *vy = a.v + a.padded + mine, *vz = a.v + 2 * a.padded + mine;
#pragma unroll
      for (int k = 0; k < kItems; ++k) {
        key[k] = kGone;
        word[k] = mine + k * kThreads;
        if (static_cast<uint32_t>(tid + k * kThreads) < home) {
          key[k] = __ldcs(keys + k * kThreads);
          f[k][0] = __ldcs(x + k * kThreads);
          f[k][1] = __ldcs(y + k * kThreads);
          f[k][2] = __ldcs(z + k * kThreads);
          f[k][3] = __ldcs(vx + k * kThreads);
          f[k][4] = __ldcs(vy + k * kThreads);
          f[k][5] = __ldcs(vz + k * kThreads);
        }
      }
    }
    const uint32_t behind = g + step;
    if (behind < groups) {
      where = tables[2 * behind];
      what = tables[2 * behind + 1];
      if (tid < 3) prefetch_range((tid == 0 ? a.x : tid == 1 ? a.y : a.z) + where.x, where.y * 4);
      else if (tid < 6) prefetch_range(a.v + (tid - 3) * a.padded + where.x, where.y * 4);
      else if (tid == 6) prefetch_range(a.keys + where.x, where.y * 4);
      else if (tid == 7) prefetch_range(a.arrived + static_cast<size_t>(where.z) * kRecordWords, where.w * 32);
    }
    const int drop = drop_for<Shape>(cells_here);
    const int dropped = max(drop, 0);
    const uint32_t drop_mask = (1u << dropped) - 1;
    const uint32_t key_base = first_cell << kShuffleBits;
    // The move; then the arrivals, which have moved already (few warps have any).
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      if (__any_sync(0xffffffffu, static_cast<uint32_t>(tid + k * kThreads) < home)) push_particle(a.push, f[k]);
      const uint32_t r = tid + k * kThreads;
      if (r >= home && r < places) {
        const uint4* arrived = reinterpret_cast<const uint4*>(a.arrived) + 2 * static_cast<size_t>(first_arrived + (r - home));
        const uint4 lo = __ldcg(arrived), hi = __ldcg(arrived + 1);
        key[k] = lo.x;
        word[k] = lo.y;
        f[k][0] = __uint_as_float(lo.z);
        f[k][1] = __uint_as_float(lo.w);
        f[k][2] = __uint_as_float(hi.x);
        f[k][3] = __uint_as_float(hi.y);
        f[k][4] = __uint_as_float(hi.z);
        f[k][5] = __uint_as_float(hi.w);
      }
    }
    barrier();  // the counters are zero

    // Written without branches around more than one access, so that the compiler predicates them.
    uint32_t run[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t low = (key[k] - key_base) >> dropped, sh = (low << 3) & 31u;
      uint32_t old = 0;
      if (key[k] != kGone) old = atomicAdd(&s.hist[low >> 2], 1u << sh);
      run[k] = (old >> sh) & 0xffu;
      word[k] |= (key[k] & drop_mask) << (32 - Shape::kMaxDrop);
    }
    barrier();

    // Exclusive scan of the counters.
    uint32_t local[kWordsPerThread];
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < kWordsPerThread; j += 4) {
      const uint4 w = *reinterpret_cast<const uint4*>(&s.hist[tid * kWordsPerThread + j]);
      local[j] = sum;
      sum = __dp4a(w.x, 0x01010101u, sum);
      local[j + 1] = sum;
      sum = __dp4a(w.y, 0x01010101u, sum);
      local[j + 2] = sum;
      sum = __dp4a(w.z, 0x01010101u, sum);
      local[j + 3] = sum;
      sum = __dp4a(w.w, 0x01010101u, sum);
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s.warp_sum[warp] = incl;
    barrier();
    // Every warp adds up the warps' sums for itself.
    const uint32_t warps = lane < kWarps ? s.warp_sum[lane] : 0u;
    const uint32_t total = __reduce_add_sync(0xffffffffu, warps);
    const uint32_t thread_base = __reduce_add_sync(0xffffffffu, lane < warp ? warps : 0u) + incl - sum;
    const uint32_t both = thread_base * 0x10001u;
#pragma unroll
    for (int j = 0; j < kWordsPerThread; j += 4) {
      uint2 prefix;  // no carry between the halves: all below 2^16
      prefix.x = both + (local[j] + (local[j + 1] << 16));
      prefix.y = both + (local[j + 2] + (local[j + 3] << 16));
      *reinterpret_cast<uint2*>(&s.word_prefix[tid * kWordsPerThread + j]) = prefix;
    }
    if (total != count) return false;  // a counter wrapped (the same answer everywhere)
    barrier();

    const int cell_words = cell_words_for(drop);
    const int hist_words = counter_words(cells_here, drop);
    for (int c = tid; c < cells_here; c += kThreads) {
      const uint32_t lo = s.word_prefix[c * cell_words];
      const uint32_t hi = (c + 1) * cell_words < hist_words ? s.word_prefix[(c + 1) * cell_words] : count;
      out.cell_start[first_cell + c] = static_cast<int32_t>(begin + lo);
      out.cell_counts[first_cell + c] = static_cast<int32_t>(hi - lo);
    }
    uint32_t longest = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t low = (key[k] != kGone ? key[k] - key_base : 0u) >> dropped, sh = (low << 3) & 31u;
      const uint32_t counters = s.hist[low >> 2];
      const uint32_t start = __dp4a(counters & ((1u << sh) - 1u), 0x01010101u, static_cast<uint32_t>(s.word_prefix[low >> 2]));
      const uint32_t length = (counters >> sh) & 0xffu;
      if (key[k] != kGone) s.tie[start + run[k]] = word[k];
      longest = max(longest, length);
      run[k] = start | length << 16;
    }
    barrier();
#pragma unroll
    for (int j = 0; j < kWordsPerThread; j += 4)
      *reinterpret_cast<uint4*>(&s.hist[tid * kWordsPerThread + j]) = make_uint4(0u, 0u, 0u, 0u);
    longest = __reduce_max_sync(0xffffffffu, longest);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t length = run[k] >> 16, start = run[k] & 0xffffu;
      const uint32_t* others = &s.tie[start];
      uint32_t slot = start;
      const uint32_t o0 = others[0], o1 = others[1], o2 = others[2];
      slot += o0 < word[k];
      slot += 1 < length && o1 < word[k];
      slot += 2 < length && o2 < word[k];
      if (longest > 3)
        for (uint32_t j = 3; j < longest; ++j)
          if (j < length) slot += others[j] < word[k];
      run[k] = slot;
    }
    barrier();
    // The places of the stage are those of the output, from the 16 bytes on in which it begins.
    const uint32_t lead = begin & 3u;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      uint32_t* to = &s.stage[0][lead + run[k]];
      if (key[k] != kGone) {
        to[0] = key[k];
        to[SettledSmem<Shape>::kRow] = word[k] & ((1u << (32 - Shape::kMaxDrop)) - 1);
#pragma unroll
        for (int c = 0; c < 6; ++c) to[(2 + c) * SettledSmem<Shape>::kRow] = __float_as_uint(f[k][c]);
      }
    }
    barrier();
    const uint32_t base = begin - lead, last = lead + count;
    for (uint32_t p = tid * 4; p < last; p += kThreads * 4) {
      uint32_t* const rows[kRecordWords] = {
          out.keys, reinterpret_cast<uint32_t*>(out.index), reinterpret_cast<uint32_t*>(out.xs),
          reinterpret_cast<uint32_t*>(out.ys), reinterpret_cast<uint32_t*>(out.zs), reinterpret_cast<uint32_t*>(out.vs),
          reinterpret_cast<uint32_t*>(out.vs + out.padded_sorted), reinterpret_cast<uint32_t*>(out.vs + 2 * out.padded_sorted)};
      if (a.vec_out && p >= lead && p + 4 <= last) {
#pragma unroll
        for (int c = 0; c < kRecordWords; ++c)
          __stcs(reinterpret_cast<uint4*>(rows[c] + (base + p)), *reinterpret_cast<const uint4*>(&s.stage[c][p]));
      } else {
#pragma unroll 1
        for (uint32_t e = max(p, lead); e < min(p + 4, last); ++e)
#pragma unroll
          for (int c = 0; c < kRecordWords; ++c) __stcs(rows[c] + (base + e), s.stage[c][e]);
      }
    }
  }
  return true;
}

template <class Shape>
__global__ void __launch_bounds__(Shape::kThreads, Shape::kBlocks)
settled_finish_kernel(const __grid_constant__ SettledArgs a, const __grid_constant__ FinishOut out) {
  // No early release: the count kernel of the general path, set up while these blocks still hold their
  // multiprocessors, would lie unevenly on them (16.8 M particles given up: 72 -> 88 us).
  chain_wait();
  const uint32_t groups = a.hdr->aux_counter[2];
  // One answer for the block: others may set the word meanwhile.
  if (__syncthreads_or(threadIdx.x == 0 && settle_failed(a.hdr))) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) out.cell_start[a.num_cells] = a.n;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  if (!finish_settled_groups(*reinterpret_cast<SettledSmem<Shape>*>(smem_raw), a, out, a.tables, blockIdx.x, groups,
                             gridDim.x, threadIdx.x, BlockBarrier{}) &&
      threadIdx.x == 0)
    fail_settle(a.hdr);
}

// The groups of dense regions, by the THREADS of the general path's finish kernel, which has nothing else to do behind a
// sort that succeeds: block `block` of `blocks`.  False if a counter wrapped.  A thread's registers are full: with two or
// three records a thread for groups of fewer, picked group by group, the compiler spilled 350 to 850 bytes and 16.8 M particles, half
// of them in a twentieth of the space, took 533 us instead of 504.
template <int THREADS>
__device__ __forceinline__ bool finish_settled_dense(unsigned char* smem, const SettledCall& call, uint32_t block,
                                                     uint32_t blocks) {
  constexpr int kPart = SettledDense::kThreads, kParts = THREADS / kPart;
  static_assert(THREADS == kParts * kPart, "whole parts");
  auto* s = reinterpret_cast<SettledSmem<SettledDense>*>(smem);
  const uint32_t* list = call.args.dense_tables;
  const uint32_t groups = call.args.hdr->aux_counter[3];
  if (block * kParts >= groups) return true;
  if constexpr (kParts == 1)
    return finish_settled_groups(*s, call.args, call.out, list, block, groups, blocks, threadIdx.x, BlockBarrier{});
  const int part = threadIdx.x / kPart;
  return finish_settled_groups(s[part], call.args, call.out, list, block * kParts + part, groups, blocks * kParts,
                               threadIdx.x % kPart, PartBarrier<kPart>{part});
}

// The records of a bucket that no block holds: its home run in the input without those that left, and its
// arrivals.
template <class Shape>
struct SettledRecords {
  const SettledArgs& a;
  uint32_t home_first, home, arrived_first, arrivals;
  template <class Use>
  __device__ __forceinline__ void keys(Use use) const {
    for (uint32_t base = 0; base < home; base += Shape::kThreads) {
      const uint32_t r = base + threadIdx.x;
      const uint32_t key = r < home ? __ldcg(a.keys + home_first + r) : kGone;
      use(key, key != kGone);
    }
    for (uint32_t base = 0; base < arrivals; base += Shape::kThreads) {
      const uint32_t r = base + threadIdx.x;
      use(r < arrivals ? __ldcg(a.arrived + static_cast<size_t>(arrived_first + r) * kRecordWords) : 0u, r < arrivals);
    }
  }
  template <class Place>
  __device__ __forceinline__ void records(Place place) const {
    for (uint32_t r = threadIdx.x; r < home; r += Shape::kThreads) {
      const int64_t i = home_first + r;
      const uint32_t key = __ldcg(a.keys + i);
      uint4* to = key != kGone ? reinterpret_cast<uint4*>(place(key)) : nullptr;
      if (!to) continue;
      float f[6] = {a.x[i], a.y[i], a.z[i], a.v[i], a.v[a.padded + i], a.v[2 * a.padded + i]};
      push_particle(a.push, f);
      to[0] = make_uint4(key, static_cast<uint32_t>(i), __float_as_uint(f[0]), __float_as_uint(f[1]));
      to[1] = make_uint4(__float_as_uint(f[2]), __float_as_uint(f[3]), __float_as_uint(f[4]), __float_as_uint(f[5]));
    }
    for (uint32_t r = threadIdx.x; r < arrivals; r += Shape::kThreads) {
      const uint4* record = reinterpret_cast<const uint4*>(a.arrived) + 2 * static_cast<size_t>(arrived_first + r);
      const uint4 lo = __ldcg(record);
      uint4* to = reinterpret_cast<uint4*>(place(lo.x));
      if (!to) continue;
      to[0] = lo;
      to[1] = __ldcg(record + 1);
    }
  }
};

// Buckets first, first + step, ... of those that no block holds.  False if one of them cannot be finished.
template <class Shape>
__device__ bool finish_settled_large(FinishSmem<Shape>& s, const SettledArgs& a, const FinishOut& out, uint32_t first,
                                     uint32_t step) {
  const uint32_t large = a.hdr->aux_counter[4];
  for (uint32_t r = first; r < large; r += step) {
    const uint4* table = reinterpret_cast<const uint4*>(a.tables) + 2 * static_cast<size_t>(a.buckets - 1 - r);
    const uint4 where = table[0], what = table[1];
    const int64_t first_cell = static_cast<int64_t>(what.z) << a.shift;
    const int cells_here = static_cast<int>(
        min(static_cast<long long>(1) << a.shift, static_cast<long long>(a.num_cells - first_cell)));
    if (!finish_large_bucket<Shape>(s, out, SettledRecords<Shape>{a, where.x, where.y, where.z, where.w}, what.x,
                                    first_cell, cells_here, [](uint32_t, int) {}))
      return false;
  }
  return true;
}
