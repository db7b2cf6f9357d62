// iq_sampling.cu -- measurement shots entirely on the device.
//
// The reference samples on the host (StateVector::sample,
// core/src/statevector.cpp:235-256): a serial cumulative distribution over
// all 2^n probabilities, std::mt19937_64 seeded with the caller's seed,
// std::uniform_real_distribution<double>(0, 1) per shot, lower_bound, clamp to
// 2^n - 1; its driver then builds the counts dictionary in Python
// (invariantq/simulator/statevector.py:105-114).  Here every step runs on the
// GPU, drawing the same random numbers so the shots are the reference's:
//
//   1. block sums of |a|^2 over blocks of 2^bb amplitudes (launch_block_sums);
//   2. their inclusive prefix (one CTA: contiguous runs per thread, then the
//      run totals in order);
//   3. the mt19937_64 stream (Matsumoto & Nishimura's 64-bit Mersenne Twister,
//      the engine the C++ standard specifies: the state of 312 words is
//      regenerated by 156 threads in two dependent halves, then tempered in
//      parallel) mapped to [0, 1) as std::generate_canonical<double, 53> does
//      for a 64-bit engine: the draw converted to double, times 2^-64, values
//      that round up to 1 replaced by the largest double below 1;
//   4. per shot a binary search for its block, then the warp search inside
//      the block (launch_block_search);
//   5. for counts: the shot indices sorted (bitonic network, in shared memory
//      where partners are near, padded to a power of two), run-length encoded
//      into ascending outcomes and their counts.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "iq_kernels.h"

namespace iqb {
namespace {

constexpr int kMtN = 312, kMtM = 156;
constexpr uint64_t kMtA = 0xB5026F5AA96619E9ULL;
constexpr uint64_t kMtUpper = 0xFFFFFFFF80000000ULL, kMtLower = 0x000000007FFFFFFFULL;

__device__ __forceinline__ uint64_t mt_mix(uint64_t cur, uint64_t nxt) {
  const uint64_t x = (cur & kMtUpper) | (nxt & kMtLower);
  return (x >> 1) ^ ((x & 1ULL) ? kMtA : 0ULL);
}

__device__ __forceinline__ uint64_t mt_temper(uint64_t z) {
  z ^= (z >> 29) & 0x5555555555555555ULL;
  z ^= (z << 17) & 0x71D67FFFEDA60000ULL;
  z ^= (z << 37) & 0xFFF7EEE000000000ULL;
  z ^= (z >> 43);
  return z;
}

// generate_canonical<double, 53> of one 64-bit draw
__device__ __forceinline__ double mt_unit(uint64_t z) {
  double r = __ull2double_rn(z) * 0x1p-64;
  if (r >= 1.0) r = 0x1.fffffffffffffp-1;
  return r;
}

// One CTA of kMtM threads: `count` uniform draws of the stream seeded with `seed`.
__global__ void __launch_bounds__(kMtM) mt64_uniform_kernel(uint64_t seed, uint64_t count, double* __restrict__ out) {
  __shared__ uint64_t mt[kMtN];
  const int t = threadIdx.x;
  if (t == 0) {   // seeding is a serial recurrence (312 steps)
    mt[0] = seed;
    for (int i = 1; i < kMtN; ++i) mt[i] = 6364136223846793005ULL * (mt[i - 1] ^ (mt[i - 1] >> 62)) + (uint64_t)i;
  }
  __syncthreads();
  for (uint64_t done = 0; done < count; done += kMtN) {
    // operands of the second half (words 156..311), read before the first half writes
    const int i2 = kMtM + t;
    const uint64_t cur2 = mt[i2];
    const uint64_t nxt2 = (i2 + 1 < kMtN) ? mt[i2 + 1] : 0ULL;
    const uint64_t new1 = mt[t + kMtM] ^ mt_mix(mt[t], mt[t + 1]);   // words 0..155: all old operands
    __syncthreads();
    mt[t] = new1;
    __syncthreads();
    // words 156..310 take word i + m - n of the new first half; word 311 also the new word 0
    const uint64_t nx = (i2 + 1 < kMtN) ? nxt2 : mt[0];
    const uint64_t new2 = mt[i2 + kMtM - kMtN] ^ mt_mix(cur2, nx);
    __syncthreads();
    mt[i2] = new2;
    __syncthreads();
    for (int j = t; j < kMtN; j += kMtM) {
      const uint64_t k = done + (uint64_t)j;
      if (k < count) out[k] = mt_unit(mt_temper(mt[j]));
    }
    __syncthreads();
  }
}

// exclusive prefix of one value per thread over a CTA of 1024 (warp scans, then
// the warp totals); *total gets the sum
template <class T>
__device__ __forceinline__ T block_exclusive(T v, T* warp_tot, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    T w = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  *total = warp_tot[31];
  return (warp ? warp_tot[warp - 1] : T(0)) + inc - v;
}

// One CTA of 1024: inclusive prefix of in[0..n) into out (contiguous runs per
// thread; the scan of the runs' sums took one thread 1024 steps before: 9.3 ->
// 3 us for one block).
__global__ void __launch_bounds__(1024) prefix_kernel(const double* __restrict__ in, uint64_t n, double* __restrict__ out) {
  __shared__ double warp_tot[32];
  const int t = threadIdx.x, T = blockDim.x;
  const uint64_t per = (n + T - 1) / T;
  const uint64_t b = (uint64_t)t * per, e = (b + per < n) ? b + per : n;
  double s = 0.0;
  for (uint64_t i = b; i < e; ++i) s += in[i];
  double total;
  double run = block_exclusive(s, warp_tot, &total);
  for (uint64_t i = b; i < e; ++i) {
    run += in[i];
    out[i] = run;
  }
}

// per shot: first block whose inclusive prefix is >= r (clamped to the last)
__global__ void find_block_kernel(const double* __restrict__ incl, uint64_t nblk, const double* __restrict__ r,
                                  int shots, uint64_t* __restrict__ blk, double* __restrict__ base) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= shots) return;
  const double x = r[k];
  uint64_t lo = 0, hi = nblk;
  while (lo < hi) {
    const uint64_t mid = lo + ((hi - lo) >> 1);
    if (incl[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  if (lo >= nblk) lo = nblk - 1;
  blk[k] = lo;
  base[k] = lo ? incl[lo - 1] : 0.0;
}

// ---- counts: the shots sorted by a bitonic network, then run-length encoded
//
// Launches bound the small cases: one per network step was 91 launches for 8192
// shots.  Steps whose partners lie within kSortTile run in shared memory, all
// of them in one launch; up to kSortTile shots the whole count is one launch.
constexpr int kSortTile = 8192;        // 64 KiB of shared memory, 1024 threads

// network steps j = j0, j0/2, .. 1 of merge size k on the tile's elements (global index base + i)
__device__ __forceinline__ void tile_steps(uint64_t* s, uint64_t base, int len, uint64_t k, int j0) {
  for (int j = j0; j > 0; j >>= 1) {
    for (int q = threadIdx.x; q < len / 2; q += blockDim.x) {
      const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), p = i | j;
      const uint64_t x = s[i], y = s[p];
      if ((x > y) == (((base + i) & k) == 0)) {
        s[i] = y;
        s[p] = x;
      }
    }
    __syncthreads();
  }
}

// tiles of in[0..n) (padded with the largest value) sorted, alternating in direction
__global__ void __launch_bounds__(1024) sort_tiles_kernel(const uint64_t* __restrict__ in, uint64_t n,
                                                          uint64_t* __restrict__ out) {
  extern __shared__ uint64_t sort_smem[];
  const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x) sort_smem[i] = base + i < n ? in[base + i] : ~0ULL;
  __syncthreads();
  for (int k = 2; k <= kSortTile; k <<= 1) tile_steps(sort_smem, base, kSortTile, (uint64_t)k, k >> 1);
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x) out[base + i] = sort_smem[i];
}

// the steps of merge size k > kSortTile whose partners lie within a tile
__global__ void __launch_bounds__(1024) merge_tiles_kernel(uint64_t* __restrict__ a, uint64_t k) {
  extern __shared__ uint64_t sort_smem[];
  const uint64_t base = (uint64_t)blockIdx.x * kSortTile;
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x) sort_smem[i] = a[base + i];
  __syncthreads();
  tile_steps(sort_smem, base, kSortTile, k, kSortTile >> 1);
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x) a[base + i] = sort_smem[i];
}

// one compare-exchange step (k, j) in global memory, one pair per thread
__global__ void bitonic_step_kernel(uint64_t* __restrict__ a, uint64_t pairs, uint64_t k, uint64_t j) {
  const uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (q >= pairs) return;
  const uint64_t i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), p = i | j;
  const uint64_t x = a[i], y = a[p];
  if ((x > y) == ((i & k) == 0)) {
    a[i] = y;
    a[p] = x;
  }
}

// a run starts at sorted position i
__device__ __forceinline__ bool run_head(const uint64_t* a, uint64_t i) { return i == 0 || a[i] != a[i - 1]; }

// One CTA, at most kSortTile shots: sort, run heads, values and counts.
__global__ void __launch_bounds__(1024) count_small_kernel(const uint64_t* __restrict__ in, int n, int npow,
                                                           uint64_t* __restrict__ vals, uint64_t* __restrict__ cnts,
                                                           uint64_t* __restrict__ nuniq) {
  extern __shared__ uint64_t sort_smem[];
  uint32_t* const pos = reinterpret_cast<uint32_t*>(sort_smem + npow);   // run heads, then n
  __shared__ uint32_t warp_tot[32];
  for (int i = threadIdx.x; i < npow; i += blockDim.x) sort_smem[i] = i < n ? in[i] : ~0ULL;
  __syncthreads();
  for (int k = 2; k <= npow; k <<= 1) tile_steps(sort_smem, 0, npow, (uint64_t)k, k >> 1);
  const int per = (n + 1023) / 1024, b = threadIdx.x * per, e = b + per < n ? b + per : n;
  uint32_t h = 0, total;
  for (int i = b; i < e; ++i) h += run_head(sort_smem, i);
  uint32_t u = block_exclusive(h, warp_tot, &total);
  for (int i = b; i < e; ++i)
    if (run_head(sort_smem, i)) {
      vals[u] = sort_smem[i];
      pos[u++] = (uint32_t)i;
    }
  if (threadIdx.x == 0) {
    pos[total] = (uint32_t)n;
    *nuniq = total;
  }
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < total; r += blockDim.x) cnts[r] = pos[r + 1] - pos[r];
}

// more shots: heads per block of 1024, their prefix, the heads' positions, the counts
__global__ void __launch_bounds__(1024) head_count_kernel(const uint64_t* __restrict__ a, uint64_t n,
                                                          uint32_t* __restrict__ blocks) {
  const uint64_t i = blockIdx.x * 1024ull + threadIdx.x;
  const int h = __syncthreads_count(i < n && run_head(a, i));
  if (threadIdx.x == 0) blocks[blockIdx.x] = (uint32_t)h;
}

__global__ void __launch_bounds__(1024) head_prefix_kernel(uint32_t* __restrict__ blocks, uint64_t nblk,
                                                           uint64_t* __restrict__ nuniq) {
  __shared__ uint32_t warp_tot[32];
  const uint64_t per = (nblk + 1023) / 1024;
  const uint64_t b = threadIdx.x * per, e = b + per < nblk ? b + per : nblk;
  uint32_t s = 0, total;
  for (uint64_t i = b; i < e; ++i) s += blocks[i];
  uint32_t run = block_exclusive(s, warp_tot, &total);
  for (uint64_t i = b; i < e; ++i) {
    const uint32_t v = blocks[i];
    blocks[i] = run;
    run += v;
  }
  if (threadIdx.x == 0) *nuniq = total;
}

__global__ void __launch_bounds__(1024) head_write_kernel(const uint64_t* __restrict__ a, uint64_t n,
                                                          const uint32_t* __restrict__ blocks,
                                                          uint64_t* __restrict__ vals, uint32_t* __restrict__ pos) {
  __shared__ uint32_t warp_tot[32];
  const uint64_t i = blockIdx.x * 1024ull + threadIdx.x;
  const bool head = i < n && run_head(a, i);
  uint32_t total;
  const uint32_t u = blocks[blockIdx.x] + block_exclusive((uint32_t)head, warp_tot, &total);
  if (head) {
    vals[u] = a[i];
    pos[u] = (uint32_t)i;
  }
}

__global__ void run_counts_kernel(const uint32_t* __restrict__ pos, const uint64_t* __restrict__ nuniq, uint64_t n,
                                  uint64_t* __restrict__ cnts) {
  const uint64_t runs = *nuniq;
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < runs; r += (uint64_t)gridDim.x * blockDim.x)
    cnts[r] = (r + 1 < runs ? pos[r + 1] : (uint32_t)n) - pos[r];
}

uint64_t sort_size(uint64_t shots) {   // power of two; whole tiles above one
  uint64_t npow = 1;
  while (npow < shots) npow <<= 1;
  return npow;
}

}  // namespace

cudaError_t launch_mt64_uniform(uint64_t seed, uint64_t count, double* out, cudaStream_t st) {
  mt64_uniform_kernel<<<1, kMtM, 0, st>>>(seed, count, out);
  return cudaGetLastError();
}

cudaError_t sample_on_device(const double2* s, int nbits, uint64_t shots, uint64_t seed, void* work, uint64_t* d_out,
                             cudaStream_t st) {
  const int bb = nbits < 12 ? nbits : 12;
  const uint64_t nblk = (1ULL << nbits) >> bb;
  double* bs = static_cast<double*>(work);
  double* incl = bs + nblk;
  double* r = incl + nblk;
  double* base = r + shots;
  uint64_t* blk = reinterpret_cast<uint64_t*>(base + shots);
  cudaError_t e = launch_block_sums(s, 1ULL << nbits, bb, bs, st);
  if (e != cudaSuccess) return e;
  prefix_kernel<<<1, 1024, 0, st>>>(bs, nblk, incl);
  mt64_uniform_kernel<<<1, kMtM, 0, st>>>(seed, shots, r);
  find_block_kernel<<<(unsigned)((shots + 255) / 256), 256, 0, st>>>(incl, nblk, r, (int)shots, blk, base);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  count_launches(5);
  return launch_block_search(s, bb, blk, base, r, d_out, (int)shots, st);
}

size_t sample_work_bytes(int nbits, uint64_t shots) {
  const int bb = std::min(12, nbits);
  const uint64_t nblk = (1ULL << nbits) >> bb;
  return (2 * nblk + 3 * shots) * 8 + 256;
}

cudaError_t count_outcomes(const uint64_t* d_shots, uint64_t shots, void* work, uint64_t* d_vals, uint64_t* d_cnts,
                           uint64_t* d_nuniq, cudaStream_t st) {
  const uint64_t npow = sort_size(shots);
  if (npow <= (uint64_t)kSortTile) {
    const size_t smem = npow * 8 + (shots + 1) * 4;
    cudaError_t e = cudaFuncSetAttribute(count_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kSortTile * 8 + (kSortTile + 1) * 4);
    if (e != cudaSuccess) return e;
    count_small_kernel<<<1, 1024, smem, st>>>(d_shots, (int)shots, (int)npow, d_vals, d_cnts, d_nuniq);
    count_launches(1);
    return cudaGetLastError();
  }
  uint64_t* a = static_cast<uint64_t*>(work);
  uint32_t* pos = reinterpret_cast<uint32_t*>(a + npow);
  uint32_t* blocks = pos + ((shots + 63) & ~(uint64_t)63);
  const size_t smem = kSortTile * 8;
  cudaError_t e = cudaFuncSetAttribute(sort_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(merge_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const unsigned tiles = (unsigned)(npow / kSortTile);
  sort_tiles_kernel<<<tiles, 1024, smem, st>>>(d_shots, shots, a);
  uint64_t launches = 1;
  for (uint64_t k = 2ull * kSortTile; k <= npow; k <<= 1) {
    for (uint64_t j = k >> 1; j >= (uint64_t)kSortTile; j >>= 1) {
      bitonic_step_kernel<<<(unsigned)(npow / 2 / 256), 256, 0, st>>>(a, npow / 2, k, j);
      ++launches;
    }
    merge_tiles_kernel<<<tiles, 1024, smem, st>>>(a, k);
    ++launches;
  }
  const uint64_t nblk = (shots + 1023) / 1024;
  head_count_kernel<<<(unsigned)nblk, 1024, 0, st>>>(a, shots, blocks);
  head_prefix_kernel<<<1, 1024, 0, st>>>(blocks, nblk, d_nuniq);
  head_write_kernel<<<(unsigned)nblk, 1024, 0, st>>>(a, shots, blocks, d_vals, pos);
  run_counts_kernel<<<(unsigned)std::min<uint64_t>(nblk, 148 * 4), 256, 0, st>>>(pos, d_nuniq, shots, d_cnts);
  count_launches(launches + 4);
  return cudaGetLastError();
}

size_t count_work_bytes(uint64_t shots) {
  const uint64_t npow = sort_size(shots);
  return npow * 8 + ((shots + 63) & ~(uint64_t)63) * 4 + ((shots + 1023) / 1024) * 4 + 256;
}

}  // namespace iqb
