// iq_ham.cu -- lambda = H psi and <psi|H|psi> for a sum H of Pauli strings, the
// middle step of an adjoint gradient and the expectation of a Pauli sum (the
// reference evaluates one string per sweep over the state,
// core/src/statevector.cpp:258-291).
//
// Strings that share their X part (a group) read the same partner amplitude:
//   lambda[x] = sum_g f_g(x) psi[x ^ xmask_g],  f_g(x) = sum_t c_t (-1)^popc(x & zmask_t).
//
// What bounds it: the partners.  Fetched from global memory, every group is
// another sweep over the state once its flips leave the caches (28 qubits: 29
// sweeps, 32.1 ms).  Here a CTA holds a tile of 2^12 amplitudes in shared
// memory -- all values of 12 chosen index bits -- so every group whose X part
// lies in those bits finds its partners there, and one sweep over the state
// serves all of them: the low 12 bits first (contiguous tiles), then 8 more
// high bits per sweep beside the 4 lowest (256-byte rows).  A sweep after the
// first adds to the lambda already stored.  Groups that fit no sweep gather
// from global memory.
//
// The sign sums f_g cost integer work per (string, amplitude).  A thread holds
// 16 amplitudes that differ in 4 tile bits only, so a string's parity splits
// into a part of the thread's own (one popc) and one of 16 patterns over those
// 4 bits: strings are sorted by pattern, summed per pattern, and a 16-point
// Walsh-Hadamard transform (4 additions per amplitude) gives f for all 16.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "iq_kernels.h"

namespace iqb {
namespace {

constexpr int kHamM = 12;              // tile bits
constexpr int kHamRegBits = 4;         // the highest tile-local bits: 16 amplitudes per thread
constexpr int kHamV = 1 << kHamRegBits;
constexpr int kHamTidBits = kHamM - kHamRegBits;
constexpr int kHamThreads = 1 << kHamTidBits;   // the other tile-local bits
constexpr int kHamChunk = 4;           // lowest index bits every tile holds

__device__ __forceinline__ double2 wide(double2 v) { return v; }
__device__ __forceinline__ double2 wide(float2 v) { return make_double2((double)v.x, (double)v.y); }
__device__ __forceinline__ void store(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void store(float2* p, double2 v) {
  *p = make_float2(__double2float_rn(v.x), __double2float_rn(v.y));
}

__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum over the block, valid in thread 0 (warps in order)
__device__ __forceinline__ double block_total(double v, double* red) {
  v = warp_total(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kHamThreads / 32; ++w) t += red[w];
  return t;
}

// Shared memory of a sweep: [tile][strings: signed coefficients, coefficients, Z and X masks][items][strings' sign
// words: one bit per thread].
// Strings past kHamSmemTerms are summed from global memory, sign by sign.
constexpr int kHamSmemTerms = 512;
constexpr int kHamStringBytes = 32 + kHamThreads / 8 + 4;
// Groups of up to this many strings add each string to the 16 sums with its own
// signs (48 instructions a string); larger ones sum per pattern and transform (64
// additions, 16 loops that few strings leave mostly empty).  One state, 60 groups
// of 3 strings with up to four flips, all by transform / these two: 14 qubits 140 /
// 90 us, 22 869 / 672; 8 strings 209 / 159, 1058 / 938; 16 to 23 strings 372 / 363,
// but 1306 / 1502 at 22.
constexpr int kHamFewStrings = 16;
constexpr int kHamLoads = 4;           // partners on their way at a time (2 and 8 spill 400 to 600 bytes)
__host__ __device__ inline int ham_smem_terms(const HamSweep& s) {
  return s.term1 - s.term0 <= kHamSmemTerms ? s.term1 - s.term0 : 0;
}
size_t ham_smem_bytes(const HamSweep& s, size_t amp) {
  return (amp << kHamM) + (size_t)ham_smem_terms(s) * kHamStringBytes + (size_t)(s.item1 - s.item0) * sizeof(HamItem);
}

// One sweep.  blockIdx.y = set: psi + set * pstride, lam + set * lstride.
// lam null: only the sums; else lambda is written (P.add 0) or added to.
// Block sums of conj(psi) times lambda -- of this sweep's share when lam is
// null, else of the stored lambda -- go to re[set * rstride + blockIdx.x] (and
// im) when re is not null.
//
// Per tile and SM at 28 qubits, TFIM, first sweep: 14 reads of the tile from
// shared memory (7200 clocks at 128 B each) against 5400 clocks of HBM traffic;
// later sweeps 9 reads (4600) against 8000.  The signs' tile part is applied to
// the coefficients once per tile and their thread part is one bit of a word
// made at the start, because a popc per (thread, string) runs at a quarter of
// the integer rate.  256 threads of 16 amplitudes: 512 threads of 8 twice the
// warps but spilled at 64 registers and read the strings twice as often (26
// qubits: 1.10 / 0.77 / 0.78 ms).  L1 at 58 %, 16 warps per SM: latency-bound.
// PLAIN: a sweep whose strings are all staged and whose items are all real, in the
// tile, and flat or of many strings (the other paths cost the chains' sweeps 2 % in
// registers).
template <class T, bool PLAIN>
__global__ void __launch_bounds__(kHamThreads, 2)
ham_sweep_kernel(const T* __restrict__ psi, uint64_t pstride, const __grid_constant__ HamSweep P,
                 const HamItem* __restrict__ g_items, const uint64_t* __restrict__ tz, const uint64_t* __restrict__ txm,
                 const double* __restrict__ tc, const ulonglong2* __restrict__ frames, T* __restrict__ lam,
                 uint64_t lstride, double* __restrict__ re, double* __restrict__ im, uint32_t rstride) {
  extern __shared__ __align__(16) unsigned char ham_smem[];
  T* const tile = reinterpret_cast<T*>(ham_smem);
  const int nterms = ham_smem_terms(P);
  double* const sc = reinterpret_cast<double*>(ham_smem + (sizeof(T) << kHamM));
  double* const c0 = sc + nterms;                      // the strings' coefficients and masks
  uint64_t* const sz = reinterpret_cast<uint64_t*>(c0 + nterms);
  uint64_t* const sx = sz + nterms;
  HamItem* const items = reinterpret_cast<HamItem*>(sx + nterms);
  uint32_t* const words = reinterpret_cast<uint32_t*>(items + (P.item1 - P.item0));
  uint32_t* const pats = words + nterms * (kHamThreads / 32);   // bit v: the string's sign at the thread's amplitude v
  __shared__ double red[kHamThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  psi += blockIdx.y * pstride;
  if (lam) lam += blockIdx.y * lstride;
  // the set's Pauli frame X^x Z^z: strings that do not commute with it change sign
  const ulonglong2 frame = frames ? frames[blockIdx.y] : make_ulonglong2(0, 0);
  auto flips = [&](uint64_t x, int k) { return (__popcll((x ^ frame.x) & tz[k]) + __popcll(txm[k] & frame.y)) & 1; };
  uint64_t tphys = 0;                  // physical bits of the thread's tile-local bits
  for (int j = 0; j < kHamTidBits; ++j)
    if ((tid >> j) & 1) tphys |= 1ULL << P.bit[j];
  uint64_t r[kHamRegBits];
  for (int j = 0; j < kHamRegBits; ++j) r[j] = 1ULL << P.bit[kHamTidBits + j];
  auto vphys = [&](int v) {
    uint64_t x = 0;
#pragma unroll
    for (int j = 0; j < kHamRegBits; ++j)
      if ((v >> j) & 1) x |= r[j];
    return x;
  };
  {
    const int words_of = (int)(sizeof(HamItem) / 4) * (P.item1 - P.item0);
    const uint32_t* src = reinterpret_cast<const uint32_t*>(g_items + P.item0);
    for (int i = tid; i < words_of; i += kHamThreads) reinterpret_cast<uint32_t*>(items)[i] = src[i];
    for (int k = tid; k < nterms; k += kHamThreads) {
      sz[k] = tz[P.term0 + k];
      sx[k] = txm[P.term0 + k];
      c0[k] = tc[P.term0 + k];
      if (PLAIN) continue;
      uint32_t m = 0;
#pragma unroll
      for (int j = 0; j < kHamRegBits; ++j) {
        constexpr uint32_t kSet[kHamRegBits] = {0xAAAAu, 0xCCCCu, 0xF0F0u, 0xFF00u};   // amplitudes with register bit j
        if ((sz[k] >> P.bit[kHamTidBits + j]) & 1) m ^= kSet[j];
      }
      pats[k] = m;
    }
    __syncthreads();
    for (int k = 0; k < nterms; ++k) {
      const uint32_t w = __ballot_sync(0xffffffffu, __popcll(tphys & sz[k]) & 1);
      if (lane == 0) words[k * (kHamThreads / 32) + warp] = w;
    }
  }
  const uint64_t dim = 1ULL << P.nbits;
  double er = 0.0, ei = 0.0;
  for (uint64_t t = blockIdx.x; t < P.ntiles; t += gridDim.x) {
    uint64_t base = t << kHamChunk;    // zeros inserted at the tile's high bits, ascending
    for (int j = kHamChunk; j < kHamM; ++j) {
      const uint64_t lo = (1ULL << P.bit[j]) - 1;
      base = ((base & ~lo) << 1) | (base & lo);
    }
    const uint64_t tx = base | tphys;
    double2 acc[kHamV];
    __syncthreads();                   // the previous tile's readers are done
#pragma unroll
    for (int v = 0; v < kHamV; ++v) {  // amplitudes past the array (fewer than 12 qubits) count as 0
      const uint64_t x = tx | vphys(v);
      T a;
      a.x = a.y = 0;
      if (x < dim) a = psi[x];
      tile[tid + v * kHamThreads] = a;
    }
#pragma unroll
    for (int v = 0; v < kHamV; ++v) {
      const uint64_t x = tx | vphys(v);
      acc[v] = (P.add && x < dim) ? wide(lam[x]) : make_double2(0.0, 0.0);
    }
    for (int k = tid; k < nterms; k += kHamThreads) {
      const bool neg = (__popcll((base ^ frame.x) & sz[k]) + __popcll(sx[k] & frame.y)) & 1;
      sc[k] = neg ? -c0[k] : c0[k];
    }
    __syncthreads();
    // sum of the strings [k0, k1) at the thread's amplitude 0
    auto strings = [&](int k0, int k1) {
      double f = 0.0;
      if (PLAIN || nterms) {
        for (int k = k0 - P.term0; k < k1 - P.term0; ++k) {
          const double c = sc[k];
          f += ((words[k * (kHamThreads / 32) + warp] >> lane) & 1) ? -c : c;
        }
      } else {
        for (int k = k0; k < k1; ++k) f += flips(tx, k) ? -tc[k] : tc[k];
      }
      return f;
    };
    for (int it = 0; it < P.item1 - P.item0; ++it) {
      const HamItem& I = items[it];
      const uint32_t flags = I.flags, mt = I.lmask & (kHamThreads - 1), mv = I.lmask / kHamThreads;
      const T* const row = tile + (tid ^ mt);
      if (PLAIN ? (flags & HAM_FLAT) != 0 : flags == HAM_FLAT) {   // real, in the tile, one f for the thread's amplitudes
        const double f = strings(I.first[0], I.first[1]);
#pragma unroll
        for (int v = 0; v < kHamV; ++v) {
          const double2 a = wide(row[(v ^ mv) * kHamThreads]);
          acc[v].x = fma(f, a.x, acc[v].x);
          acc[v].y = fma(f, a.y, acc[v].y);
        }
        continue;
      }
      double f[kHamV];
      if (!PLAIN && (flags & HAM_FLAT)) {
        const double f0 = strings(I.first[0], I.first[1]);
#pragma unroll
        for (int v = 0; v < kHamV; ++v) f[v] = f0;
      } else if (!PLAIN && nterms && I.first[kHamV] - I.first[0] <= kHamFewStrings) {
#pragma unroll
        for (int v = 0; v < kHamV; ++v) f[v] = 0.0;
        for (int k = I.first[0] - P.term0; k < I.first[kHamV] - P.term0; ++k) {
          const int hi = __double2hiint(sc[k]), lo = __double2loint(sc[k]);
          const uint32_t neg = pats[k] ^ (((words[k * (kHamThreads / 32) + warp] >> lane) & 1) ? 0xFFFFu : 0u);
#pragma unroll
          for (int v = 0; v < kHamV; ++v)
            f[v] += __hiloint2double(hi ^ (int)((neg << (31 - v)) & 0x80000000u), lo);
        }
      } else {
#pragma unroll
        for (int p = 0; p < kHamV; ++p) f[p] = strings(I.first[p], I.first[p + 1]);
#pragma unroll
        for (int h = 1; h < kHamV; h <<= 1)
#pragma unroll
          for (int v = 0; v < kHamV; ++v)
            if (!(v & h)) {
              const double a = f[v], b = f[v | h];
              f[v] = a + b;
              f[v | h] = a - b;
            }
      }
      if (PLAIN || !(flags & (HAM_GATHER | HAM_IMAG))) {
#pragma unroll
        for (int v = 0; v < kHamV; ++v) {
          const double2 a = wide(row[(v ^ mv) * kHamThreads]);
          acc[v].x = fma(f[v], a.x, acc[v].x);
          acc[v].y = fma(f[v], a.y, acc[v].y);
        }
        continue;
      }
      const uint64_t gx = tx ^ I.xmask;
      const bool gather = flags & HAM_GATHER, imag = flags & HAM_IMAG;
#pragma unroll
      for (int v0 = 0; v0 < kHamV; v0 += kHamLoads) {
        double2 a[kHamLoads];
#pragma unroll
        for (int v = 0; v < kHamLoads; ++v) {
          const uint64_t x = gx ^ vphys(v0 + v);
          a[v] = make_double2(0.0, 0.0);
          if (!gather) a[v] = wide(row[((v0 + v) ^ mv) * kHamThreads]);
          else if (x < dim) a[v] = wide(psi[x]);
        }
#pragma unroll
        for (int v = 0; v < kHamLoads; ++v) {
          const double2 t = imag ? make_double2(-a[v].y, a[v].x) : a[v];   // times i
          acc[v0 + v].x = fma(f[v0 + v], t.x, acc[v0 + v].x);
          acc[v0 + v].y = fma(f[v0 + v], t.y, acc[v0 + v].y);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < kHamV; ++v) {
      const uint64_t x = tx | vphys(v);
      if (re) {
        const double2 a = wide(tile[tid + v * kHamThreads]);
        er += a.x * acc[v].x + a.y * acc[v].y;
        if (im) ei += a.x * acc[v].y - a.y * acc[v].x;
      }
      if (lam && x < dim) store(lam + x, acc[v]);
    }
  }
  if (re) {
    er = block_total(er, red);
    ei = block_total(ei, red);
    if (tid == 0) {
      re[(size_t)blockIdx.y * rstride + blockIdx.x] = er;
      if (im) im[(size_t)blockIdx.y * rstride + blockIdx.x] = ei;
    }
  }
}

// The sum with one amplitude per thread, partners from global memory (sweeps[0]
// of a plan of one sweep holds every item).  Arrays of few tiles leave most SMs
// without one, and a group costs its tile ~1 us of a serial chain; here the array
// is spread over every SM and a group costs a sweep over it.  gather_pays has the
// line between the two.
constexpr int kGatherThreads = 256;
static_assert(kRedBlocks <= kHamPartials, "a gather launch has a partial sum per block");
constexpr int kGatherStrings = 2048;   // staged at a time
template <class T>
__global__ void __launch_bounds__(kGatherThreads)
ham_gather_kernel(const T* __restrict__ psi, uint64_t pstride, const __grid_constant__ HamSweep P,
                  const HamItem* __restrict__ g_items, const uint64_t* __restrict__ tz, const uint64_t* __restrict__ txm,
                  const double* __restrict__ tc, const ulonglong2* __restrict__ frames, T* __restrict__ lam,
                  uint64_t lstride, double* __restrict__ re, double* __restrict__ im, uint32_t rstride) {
  struct Group { uint64_t xmask; int first, last; };   // last: bit 30 marks imaginary coefficients
  __shared__ Group groups[2 * kMaxHamGroups];
  __shared__ ulonglong2 strings[kGatherStrings];       // Z mask; coefficient with the sign of the set's Pauli frame
  __shared__ double red[kHamThreads / 32];
  const int tid = threadIdx.x, ng = P.item1 - P.item0, nt = P.term1 - P.term0;
  const int chunks = (nt + kGatherStrings - 1) / kGatherStrings;
  const ulonglong2 frame = frames ? frames[blockIdx.y] : make_ulonglong2(0, 0);
  psi += blockIdx.y * pstride;
  if (lam) lam += blockIdx.y * lstride;
  for (int i = tid; i < ng; i += kGatherThreads) {
    const HamItem& I = g_items[P.item0 + i];
    groups[i] = {I.xmask, I.first[0] - P.term0, (I.first[kHamV] - P.term0) | ((I.flags & HAM_IMAG) ? 1 << 30 : 0)};
  }
  auto stage = [&](int chunk) {
    for (int k = chunk * kGatherStrings + tid; k < min(nt, (chunk + 1) * kGatherStrings); k += kGatherThreads) {
      const uint64_t z = tz[P.term0 + k];
      const double c = tc[P.term0 + k];
      const bool neg = (__popcll(frame.x & z) + __popcll(txm[P.term0 + k] & frame.y)) & 1;
      strings[k - chunk * kGatherStrings] = make_ulonglong2(z, (uint64_t)__double_as_longlong(neg ? -c : c));
    }
  };
  if (chunks == 1) stage(0);
  __syncthreads();
  const uint64_t dim = 1ULL << P.nbits;
  double er = 0.0, ei = 0.0;
  for (uint64_t x0 = blockIdx.x * (uint64_t)kGatherThreads; x0 < dim; x0 += (uint64_t)gridDim.x * kGatherThreads) {
    const uint64_t x = x0 + tid;
    const bool on = x < dim;
    double2 acc = make_double2(0.0, 0.0);
    for (int ch = 0; ch < chunks; ++ch) {
      if (chunks > 1) {
        __syncthreads();
        stage(ch);
        __syncthreads();
      }
      if (!on) continue;
      const int k0 = ch * kGatherStrings, k1 = k0 + kGatherStrings;
      double2 next = wide(psi[x ^ groups[0].xmask]);
      for (int g = 0; g < ng; ++g) {
        double2 a = next;
        if (g + 1 < ng && groups[g + 1].xmask != groups[g].xmask)
          next = wide(psi[x ^ groups[g + 1].xmask]);   // on its way during the signs
        const int first = max(groups[g].first, k0), last = min(groups[g].last & ((1 << 30) - 1), k1);
        if (first >= last) continue;
        double f = 0.0;
        for (int k = first; k < last; ++k) {
          const ulonglong2 s = strings[k - k0];
          const double c = __longlong_as_double((long long)s.y);
          f += (__popcll(x & s.x) & 1) ? -c : c;
        }
        if (groups[g].last >> 30) a = make_double2(-a.y, a.x);   // times i
        acc.x = fma(f, a.x, acc.x);
        acc.y = fma(f, a.y, acc.y);
      }
    }
    if (!on) continue;
    if (lam) store(lam + x, acc);
    const double2 px = wide(psi[x]);
    er += px.x * acc.x + px.y * acc.y;
    ei += px.x * acc.y - px.y * acc.x;
  }
  er = block_total(er, red);
  if (im) ei = block_total(ei, red);
  if (tid == 0) {
    re[(size_t)blockIdx.y * rstride + blockIdx.x] = er;
    if (im) im[(size_t)blockIdx.y * rstride + blockIdx.x] = ei;
  }
}

// the largest sweep: 64 groups of two items, kHamSmemTerms strings
template <class T>
constexpr size_t ham_smem_limit() {
  return (sizeof(T) << kHamM) + (size_t)kHamSmemTerms * kHamStringBytes + 2 * kMaxHamGroups * sizeof(HamItem);
}

template <class T>
cudaError_t run_sweeps(const HamPlan& hp, const HamTables& tb, const ulonglong2* frames, const T* psi,
                       uint64_t pstride, int nsets, T* lam, uint64_t lstride, double* partials, double* energy, double* energy_im, cudaStream_t st) {
  if (nsets < 1) nsets = 1;
  if (hp.gather) {
    const HamSweep& s = hp.sweeps[0];
    const uint32_t grid = (uint32_t)std::min<uint64_t>(((1ULL << s.nbits) + kGatherThreads - 1) / kGatherThreads, kRedBlocks);
    double* const im = energy_im ? partials + (size_t)nsets * grid : nullptr;
    ham_gather_kernel<T><<<dim3(grid, nsets), kGatherThreads, 0, st>>>(psi, pstride, s, tb.items, tb.z, tb.x, tb.c, frames, lam,
                                                                      lstride, partials, im, grid);
    cudaError_t e = launch_row_sums(partials, nsets, (int)grid, energy, st);
    if (e == cudaSuccess && energy_im) e = launch_row_sums(im, nsets, (int)grid, energy_im, st);
    return e;
  }
  size_t smem_max = 0;
  for (const HamSweep& w : hp.sweeps) smem_max = std::max(smem_max, ham_smem_bytes(w, sizeof(T)));
  // per device, so on every call (always the same value: threads may race on it)
  cudaError_t attr = cudaFuncSetAttribute(ham_sweep_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)ham_smem_limit<T>());
  if (attr == cudaSuccess)
    attr = cudaFuncSetAttribute(ham_sweep_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)ham_smem_limit<T>());
  if (attr != cudaSuccess) return attr;
  if (smem_max > ham_smem_limit<T>()) return cudaErrorInvalidValue;
  // sums: one column per block; every sweep's when lambda is not kept, else the last one's
  const int np = (int)hp.sweeps.size();
  const int cols = lam ? 1 : np;
  const uint32_t grid = (uint32_t)std::min<uint64_t>(hp.sweeps[0].ntiles, kHamBlocks);
  const uint32_t rstride = grid * (uint32_t)cols;
  double* const im = energy_im ? partials + (size_t)nsets * rstride : nullptr;
  for (int i = 0; i < np; ++i) {
    HamSweep s = hp.sweeps[i];
    s.add = (lam && i > 0) ? 1 : 0;
    const bool sums = !lam || i == np - 1;
    const size_t at = lam ? 0 : (size_t)i * grid;
    bool plain = ham_smem_terms(s) > 0;
    for (int it = s.item0; it < s.item1; ++it) {
      const HamItem& I = hp.items[it];
      plain = plain && !(I.flags & (HAM_GATHER | HAM_IMAG)) &&
              ((I.flags & HAM_FLAT) || I.first[kHamV] - I.first[0] > kHamFewStrings);
    }
    (plain ? ham_sweep_kernel<T, true> : ham_sweep_kernel<T, false>)<<<dim3(grid, nsets), kHamThreads, ham_smem_bytes(s, sizeof(T)), st>>>(
        psi, pstride, s, tb.items, tb.z, tb.x, tb.c, frames, lam, lstride, sums ? partials + at : nullptr,
        (sums && im) ? im + at : nullptr, rstride);
  }
  cudaError_t e = launch_row_sums(partials, nsets, (int)rstride, energy, st);
  if (e == cudaSuccess && energy_im) e = launch_row_sums(im, nsets, (int)rstride, energy_im, st);
  return e;
}

}  // namespace

// Whether one amplitude per thread is the faster form for a plan's sweeps.  Its
// time (us) follows groups and strings and the array past 2^16 amplitudes, where
// every SM is busy; the sweeps' is a chain of groups per tile, the same for every
// array of up to as many tiles as fit the GPU at once.  Both sides measured, one
// state, sweeps / gather: TFIM 13 qubits 22.2 / 11.5, 18 34.4 / 28.8, 20 43 / 82;
// 60 groups of 3 strings with up to four flips 87 / 24, 124 / 78, 166 / 248; 400
// diagonal strings 47 / 22, 47 / 78, 54 / 249; 16 states of 14 qubits 31 / 22, 91 /
// 64, 47 / 66.
static bool gather_pays(const HamPlan& hp, int n, int nsets) {
  const double amps = std::ldexp((double)std::max(1, nsets), n);
  double tiles = 8.0 + 2.0 * (double)hp.sweeps.size(), groups = 0.0;
  for (size_t i = 0; i < hp.items.size(); ++i) {
    const HamItem& I = hp.items[i];
    const double k = I.first[kHamV] - I.first[0];
    tiles += (I.flags & HAM_FLAT) ? 0.5 + std::min(0.2 * k, 3.0 + 0.1 * k) : std::min(0.8 + 0.3 * k, 4.0 + 0.1 * k);
    if (I.flags & HAM_GATHER) tiles += 0.8;
    groups += i && I.xmask == hp.items[i - 1].xmask ? 0.25 : 1.0;   // a group's imaginary part reads the same partner
  }
  const double gather = 8.0 + std::max(1.0, amps / 65536.0) * (0.2 * groups + 0.04 * (double)hp.z.size());
  return gather < tiles * std::max(1.0, amps / ((double)kHamBlocks * (1 << kHamM)));
}

static void plan_sweeps(int n, const HamTerms& h, const uint64_t* zmask, const double2* coef, int max_sweeps, HamPlan& hp);

void plan_hamiltonian(int n, const HamTerms& h, const uint64_t* zmask, const double2* coef, int max_sweeps, int nsets,
                      HamPlan& hp) {
  plan_sweeps(n, h, zmask, coef, max_sweeps, hp);
  const char* form = getenv("IQ_HAM_GATHER");   // 0, 1: this form whatever the sizes
  hp.gather = form && *form ? atoi(form) != 0 : gather_pays(hp, n, nsets);
  if (hp.gather && hp.sweeps.size() > 1) plan_sweeps(n, h, zmask, coef, 1, hp);
}

static void plan_sweeps(int n, const HamTerms& h, const uint64_t* zmask, const double2* coef, int max_sweeps, HamPlan& hp) {
  hp.sweeps.clear();
  hp.items.clear();
  hp.z.clear();
  hp.x.clear();
  hp.c.clear();
  const uint64_t low = (1ULL << kHamChunk) - 1;
  std::vector<uint8_t> done(h.ngroups, 0);
  for (int s = 0;; ++s) {
    // the sweep's index bits: the low 12, or the chunk and the high bits of the groups not served yet
    uint64_t local = s == 0 ? (1ULL << kHamM) - 1 : low;
    std::vector<int> mine;
    const bool last = s == max_sweeps - 1;
    for (int g = 0; g < h.ngroups; ++g) {
      if (done[g]) continue;
      const uint64_t want = local | h.xmask[g];
      if (s == 0 ? want == local : __builtin_popcountll(want) <= kHamM) {
        local = want;
        mine.push_back(g);
        done[g] = 1;
      }
    }
    // what no sweep will hold gathers in this one: groups wider than a tile in the first, all others in the last allowed
    std::vector<int> far;
    for (int g = 0; g < h.ngroups; ++g)
      if (!done[g] && (last || (s == 0 && __builtin_popcountll(low | h.xmask[g]) > kHamM))) {
        far.push_back(g);
        done[g] = 1;
      }
    for (int b = kHamChunk; __builtin_popcountll(local) < kHamM; ++b) local |= 1ULL << b;   // pad with low bits
    HamSweep w{};
    w.nbits = n;
    w.item0 = (int)hp.items.size();
    w.term0 = (int)hp.z.size();
    w.ntiles = n > kHamM ? 1ULL << (n - kHamM) : 1;
    uint64_t at[64];                   // tile-local bit of a physical bit
    int j = 0;
    for (int b = 0; b < 64; ++b)
      if ((local >> b) & 1) {
        w.bit[j] = (uint8_t)b;
        at[b] = j++;
      }
    auto add_group = [&](int g, bool gather) {
      uint32_t lm = 0;
      if (!gather)
        for (int b = 0; b < 64; ++b)
          if ((h.xmask[g] >> b) & 1) lm |= 1u << at[b];
      for (int part = 0; part < 2; ++part) {
        HamItem I{};
        I.xmask = h.xmask[g];
        I.lmask = lm;
        I.flags = (gather ? HAM_GATHER : 0) | (part ? HAM_IMAG : 0) | HAM_FLAT;
        I.first[0] = (int)hp.z.size();
        for (int p = 0; p < kHamV; ++p) {
          for (int t = h.first[g]; t < h.first[g + 1]; ++t) {
            const double c = part ? coef[t].y : coef[t].x;
            // a zero coefficient still multiplies its amplitudes once (a NaN among them shows in the result)
            if (c == 0.0 && (part || coef[t].y != 0.0)) continue;
            int pat = 0;
            for (int i = 0; i < kHamRegBits; ++i) pat |= (int)((zmask[t] >> w.bit[kHamTidBits + i]) & 1) << i;
            if (pat != p) continue;
            if (p) I.flags &= ~HAM_FLAT;
            hp.z.push_back(zmask[t]);
            hp.x.push_back(h.xmask[g]);
            // the sign is that of the partner index x ^ xmask
            hp.c.push_back((__builtin_popcountll(h.xmask[g] & zmask[t]) & 1) ? -c : c);
          }
          I.first[p + 1] = (int)hp.z.size();
        }
        if (I.first[kHamV] > I.first[0]) hp.items.push_back(I);
      }
    };
    for (int g : mine) add_group(g, false);
    for (int g : far) add_group(g, true);
    w.item1 = (int)hp.items.size();
    w.term1 = (int)hp.z.size();
    hp.sweeps.push_back(w);
    bool left = false;
    for (int g = 0; g < h.ngroups; ++g) left |= !done[g];
    if (!left) return;
  }
}

size_t HamPlan::table_bytes() const {
  return items.size() * sizeof(HamItem) + (z.size() + x.size()) * sizeof(uint64_t) + c.size() * sizeof(double);
}

void HamPlan::pack(void* dst) const {
  char* p = static_cast<char*>(dst);
  std::memcpy(p, items.data(), items.size() * sizeof(HamItem));
  p += items.size() * sizeof(HamItem);
  std::memcpy(p, z.data(), z.size() * sizeof(uint64_t));
  p += z.size() * sizeof(uint64_t);
  std::memcpy(p, x.data(), x.size() * sizeof(uint64_t));
  p += x.size() * sizeof(uint64_t);
  std::memcpy(p, c.data(), c.size() * sizeof(double));
}

HamTables HamPlan::tables(const void* dev) const {
  const char* p = static_cast<const char*>(dev);
  HamTables t;
  t.items = reinterpret_cast<const HamItem*>(p);
  p += items.size() * sizeof(HamItem);
  t.z = reinterpret_cast<const uint64_t*>(p);
  p += z.size() * sizeof(uint64_t);
  t.x = reinterpret_cast<const uint64_t*>(p);
  p += x.size() * sizeof(uint64_t);
  t.c = reinterpret_cast<const double*>(p);
  return t;
}

cudaError_t launch_hamiltonian(const HamPlan& hp, const HamTables& tb, const ulonglong2* frames, const double2* psi,
                               uint64_t pstride, int nsets, double2* lam, uint64_t lstride, double* partials, double* energy, double* energy_im,
                               cudaStream_t st) {
  return run_sweeps(hp, tb, frames, psi, pstride, nsets, lam, lstride, partials, energy, energy_im, st);
}

cudaError_t launch_hamiltonian_c64(const HamPlan& hp, const HamTables& tb, const ulonglong2* frames, const float2* psi,
                                   uint64_t pstride, int nsets, float2* lam, uint64_t lstride, double* partials, double* energy,
                                   cudaStream_t st) {
  return run_sweeps(hp, tb, frames, psi, pstride, nsets, lam, lstride, partials, energy, (double*)nullptr, st);
}

}  // namespace iqb
