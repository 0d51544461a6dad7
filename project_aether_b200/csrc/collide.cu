// No-Time-Counter collisions on cell-sorted particles for sm_100a.
//
// Replaces the reference's sm_90a kernel (custom_kernels/cuda/dsmc_collide_tma.cu:
// one warp per cell, 2-D TMA boxes of a fixed window, a second kernel for large
// cells) behind the same C entry point (dsmc_collide_tma.h:121-129).  The
// arithmetic of a pair follows dsmc_collide_tma.h:59-113 with every product and
// sum rounded on its own, as the reference's host replay computes them
// (dsmc_collide_tma_test.cu:45-84).
//
// Layout of the work: a block owns a run of consecutive cells, at most one per thread.  It draws every
// cell's number of candidate pairs, scans the numbers, and hands the pairs of ALL its cells out
// to its threads one pair per thread, so that cells of ten particles keep a block as busy as
// cells of a thousand.  A pair's velocities are read from and, if it collides, written to
// global memory directly: pair p of a cell is its particles 2p and 2p + 1, so neighbouring
// threads read neighbouring words, no two pairs share a particle, and the sectors of the many
// particles that are in no candidate pair are neither read nor written.
#include <algorithm>

#include "common.cuh"

namespace aether {
namespace {

constexpr int kCollideThreads = 256;
constexpr int kCollideBlocks = 6;               // per multiprocessor
constexpr uint32_t kCellDraw = 0xFFFFFFFFu;     // pair id of a cell's selection draw

struct CollideArgs {
  float* velocity;
  const int* cell_start;
  float* sigma_g_max;
  int* collisions;
  int padded;
  int num_cells;
  int cells_per_block;  // at most kCollideThreads
  float selection_factor, coefficient, exponent;
  uint32_t key0, key1, step_lo, step_hi;
};

// Philox4x32-10, all four words (cuda/philox.h:56-72).
__device__ __forceinline__ uint4 philox4(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                         uint32_t k0, uint32_t k1) {
  constexpr uint32_t kM0 = 0xD2511F53u, kM1 = 0xCD9E8D57u;
  constexpr uint32_t kW0 = 0x9E3779B9u, kW1 = 0xBB67AE85u;
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
  return make_uint4(c0, c1, c2, c3);
}

// 24 random bits as a float in [0, 1) (cuda/philox.h:77-79).
__device__ __forceinline__ float unit_float(uint32_t bits) {
  return __fmul_rn(static_cast<float>(bits >> 8), 1.0f / 16777216.0f);
}

__device__ __forceinline__ uint4 collision_words(int cell, uint32_t pair, const CollideArgs& a) {
  return philox4(static_cast<uint32_t>(cell), pair, a.step_lo, a.step_hi, a.key0, a.key1);
}

// floor(1/2 N (N-1) F sigma_g_max + U), at most N/2 (dsmc_collide_tma.h:63-72).
__device__ __forceinline__ int ntc_selections(int count, float majorant, float factor, float u) {
  float expected = __fmul_rn(0.5f, static_cast<float>(count));
  expected = __fmul_rn(expected, static_cast<float>(count - 1));
  expected = __fmul_rn(expected, factor);
  expected = __fmul_rn(expected, majorant);
  const int selections = static_cast<int>(floorf(__fadd_rn(expected, u)));
  return min(selections, count / 2);
}

// Tests one candidate pair and scatters it isotropically in the centre-of-mass
// frame when it is accepted (dsmc_collide_tma.h:89-113).
__device__ __forceinline__ bool collide_pair(float* a, float* b, float majorant,
                                             const CollideArgs& p, const uint4& r,
                                             float* sigma_g) {
  const float gx = __fsub_rn(a[0], b[0]), gy = __fsub_rn(a[1], b[1]), gz = __fsub_rn(a[2], b[2]);
  const float g = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)), __fmul_rn(gz, gz)));
  *sigma_g = g > 0.0f ? __fmul_rn(p.coefficient, powf(g, p.exponent)) : 0.0f;
  if (__fmul_rn(unit_float(r.x), majorant) >= *sigma_g) return false;
  const float cos_chi = __fsub_rn(__fmul_rn(2.0f, unit_float(r.y)), 1.0f);
  const float sin_chi = sqrtf(fmaxf(__fsub_rn(1.0f, __fmul_rn(cos_chi, cos_chi)), 0.0f));
  const float azimuth = __fmul_rn(6.28318530718f, unit_float(r.z));
  const float gs = __fmul_rn(g, sin_chi);
  const float post[3] = {__fmul_rn(gs, cosf(azimuth)), __fmul_rn(gs, sinf(azimuth)),
                         __fmul_rn(g, cos_chi)};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float center = __fmul_rn(0.5f, __fadd_rn(a[c], b[c]));
    const float half = __fmul_rn(0.5f, post[c]);
    a[c] = __fadd_rn(center, half);
    b[c] = __fsub_rn(center, half);
  }
  return true;
}

// Bound by the latency of a block's chain (starts, draw, scan, pairs, results) and by the sectors
// that hold candidate pairs; so little shared memory, and six blocks of 256 threads (40
// registers) per multiprocessor.  A first design staged every particle of the block's cells in
// shared memory, four blocks per multiprocessor, and wrote the stage back: 16 M particles in 2 M
// cells took it 123 us, this kernel 61 (436 MB if every velocity is read and written once).  Chained to the kernel before
// it, the sort's last in a step: step of 100,000 particles 30.2 -> 27.4 us, of 200,003 33.3 -> 31.7, of 1 M 57.8 -> 55.5,
// of 16.8 M 441 -> 438.
__global__ void __launch_bounds__(kCollideThreads, kCollideBlocks)
collide_kernel(CollideArgs a) {
  __shared__ int start[kCollideThreads];
  __shared__ int pair_first[kCollideThreads];      // exclusive prefix of the candidate pairs
  __shared__ int accepted[kCollideThreads];
  __shared__ uint32_t observed[kCollideThreads];   // largest sigma*g seen, as float bits (non-negative)
  __shared__ float majorants[kCollideThreads];     // sigma_g_max before this step
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t total;
  const int tid = threadIdx.x;
  const int first_cell = blockIdx.x * a.cells_per_block;
  const int cells_here = min(a.cells_per_block, a.num_cells - first_cell);
  const int my_cell = first_cell + tid;
  float majorant = 0.0f;
  uint32_t selections = 0;
  // Set up, and its cells' numbers drawn, while the kernel before it ends.
  const float drawn = unit_float(collision_words(my_cell, kCellDraw, a).x);
  chain_wait();
  if (tid < cells_here) {
    const int begin = a.cell_start[my_cell];
    const int count = a.cell_start[my_cell + 1] - begin;
    majorant = a.sigma_g_max[my_cell];
    selections = static_cast<uint32_t>(max(
        0, ntc_selections(count, majorant, a.selection_factor, drawn)));
    start[tid] = begin;
    accepted[tid] = 0;
    observed[tid] = 0;
    majorants[tid] = majorant;
  }
  const int before = static_cast<int>(block_exclusive_scan(selections, warp_sum, &total));
  pair_first[tid] = before;
  __syncthreads();
  const int pairs = static_cast<int>(total);
  for (int p = tid; p < pairs; p += kCollideThreads) {
    // The cell of pair p: last t with pair_first[t] <= p (cells without pairs share a value).
    int t = 0;
#pragma unroll
    for (int step = kCollideThreads / 2; step > 0; step >>= 1)
      if (pair_first[t + step] <= p) t += step;
    const uint32_t pair = static_cast<uint32_t>(p - pair_first[t]);
    const size_t i = static_cast<size_t>(start[t]) + 2 * pair;
    float v1[3], v2[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v1[c] = a.velocity[static_cast<size_t>(c) * a.padded + i];
      v2[c] = a.velocity[static_cast<size_t>(c) * a.padded + i + 1];
    }
    float sigma_g = 0.0f;
    if (collide_pair(v1, v2, majorants[t], a, collision_words(first_cell + t, pair, a), &sigma_g)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        a.velocity[static_cast<size_t>(c) * a.padded + i] = v1[c];
        a.velocity[static_cast<size_t>(c) * a.padded + i + 1] = v2[c];
      }
      atomicAdd(&accepted[t], 1);
    }
    if (sigma_g > 0.0f) atomicMax(&observed[t], __float_as_uint(sigma_g));
  }
  __syncthreads();
  if (tid < cells_here) {
    const float raised = fmaxf(majorant, __uint_as_float(observed[tid]));
    if (__float_as_uint(raised) != __float_as_uint(majorant)) a.sigma_g_max[my_cell] = raised;
    a.collisions[my_cell] = accepted[tid];
  }
}

// Cells per block: as many as a block has threads, fewer (halved, at least 16) until there is a
// block for every place on the multiprocessors, six each; a block's threads share the pairs of
// its cells whatever their number, but a block with few cells wastes threads on the cells' own
// work.  0.075 pairs per particle, 256 cells per block / this rule: 10,000 cells of 400 particles
// 46 / 13 us, 1000 cells of 400 45 / 10, 65,536 cells of 61 12.8 / 12.3; 128 cells per block at
// 2 M cells of 8 take 76 us against 62.
constexpr int kFewestCells = 16;
int cells_per_block_for(int num_cells) {
  const int places = kCollideBlocks * sm_count();
  int cells = kCollideThreads;
  while (cells > kFewestCells && (num_cells + cells - 1) / cells < places) cells /= 2;
  return cells;
}

}  // namespace

// Enqueues one collision step.  velocity (3, padded) is updated in place,
// sigma_g_max (C,) is raised to the largest sigma*g observed, collisions (C,)
// receives the accepted pairs of every cell.
cudaError_t collide_cells(float* velocity, const int* cell_start, float* sigma_g_max,
                          int* collisions, int num_particles, int padded, int num_cells,
                          float selection_factor, float coefficient, float exponent,
                          uint64_t seed, uint64_t step, cudaStream_t stream) {
  if (num_particles < 0 || num_cells < 0 || padded < num_particles || padded % 4 != 0)
    return cudaErrorInvalidValue;
  if (num_cells == 0) return cudaSuccess;
  if (!velocity || !cell_start || !sigma_g_max || !collisions) return cudaErrorInvalidValue;
  CollideArgs a{};
  a.velocity = velocity;
  a.cell_start = cell_start;
  a.sigma_g_max = sigma_g_max;
  a.collisions = collisions;
  a.padded = padded;
  a.num_cells = num_cells;
  a.selection_factor = selection_factor;
  a.coefficient = coefficient;
  a.exponent = exponent;
  a.key0 = static_cast<uint32_t>(seed);
  a.key1 = static_cast<uint32_t>(seed >> 32);
  a.step_lo = static_cast<uint32_t>(step);
  a.step_hi = static_cast<uint32_t>(step >> 32);
  a.cells_per_block = cells_per_block_for(num_cells);
  const int blocks = (num_cells + a.cells_per_block - 1) / a.cells_per_block;
  stage_begin(kStageCollide, stream);
  const cudaError_t e = launch_chained(collide_kernel, blocks, kCollideThreads, 0, stream, a);
  stage_end(kStageCollide, stream);
  count_launches(1);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace aether
