// iq_entropy.cu -- the spectrum of a reduced state, on the GPU, for the
// entanglement entropy of a state vector across a cut (the reference computes
// it in StateVector::entanglement_entropy, core/src/statevector.cpp:293-410,
// with a capped Jacobi iteration on the host; its drivers call it on every run
// for the half cut range(n // 2), invariantq/simulator/statevector.py:87-90).
//
// For a kept qubit set K (|K| = k, kd = 2^k) and the traced set E (ed = 2^(n-k)):
//
//   1. Gram kernel: rho[r][c] = sum_e psi[dep_K(r) | dep_E(e)] conj(psi[dep_K(c) | dep_E(e)]),
//      an FP64 complex rank-ed Hermitian product (rho = M M^H for the kd x ed
//      matrix M of the reshaped state), tiled 64 x 64 per CTA through shared
//      memory, upper-triangle tiles only, with the environment split across
//      CTAs in fixed chunks (deterministic: partial tiles summed in order).
//   2. Householder reduction of rho to real symmetric tridiagonal form on the
//      device: one cooperative launch up to 4096 (one barrier per column), four
//      launches per column above.
//   3. Eigenvalues of the tridiagonal matrix by multisection on Sturm counts,
//      one warp per eigenvalue.
//
// Bit i of the kept index r is qubit keep[i]; the spectrum does not depend on
// the order.  Only the eigenvalues (kd doubles) come back to the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstdint>
#include <vector>

#include "iq_kernels.h"

namespace iqb {
namespace {

constexpr int kGT = 64;        // Gram tile (rows and columns)
constexpr int kGK = 16;        // environment entries per shared-memory step
constexpr int kGThreads = 256;

// block-wide sum, result in every thread
__device__ double block_allsum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  return t;
}

// index of environment entry e: dep_E(e) = lo[e & lomask] | hi[e >> lobits]
struct EnvDep {
  const uint64_t* lo;
  const uint64_t* hi;
  int lobits;
};

__device__ __forceinline__ uint64_t env_index(const EnvDep& d, uint64_t e) {
  return d.lo[e & ((1ULL << d.lobits) - 1)] | d.hi[e >> d.lobits];
}

// grid.x = upper-triangle tile pairs (tr <= tc), grid.y = environment split s.
// part[s][tile][64 x 64] for nsplit > 1, else written straight into rho.
__global__ void __launch_bounds__(kGThreads) gram_kernel(const double2* __restrict__ psi,
                                                         const uint64_t* __restrict__ depk, EnvDep dep, int tiles,
                                                         uint64_t kd, uint64_t env_per_split,
                                                         double2* __restrict__ part, double2* __restrict__ rho) {
  __shared__ double2 As[kGK][kGT];
  __shared__ double2 Bs[kGK][kGT];
  // decode the tile pair
  int tr = 0, rem = blockIdx.x;
  while (rem >= tiles - tr) {
    rem -= tiles - tr;
    ++tr;
  }
  const int tc = tr + rem;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const uint64_t e_begin = (uint64_t)blockIdx.y * env_per_split, e_end = e_begin + env_per_split;
  // loader coordinates: row rl of the tile, environment entries el, el + 4, el + 8, el + 12
  const int rl = tid & 63, el = tid >> 6;
  const uint64_t ra = (uint64_t)tr * kGT + rl, rb = (uint64_t)tc * kGT + rl;
  const uint64_t ia = (ra < kd) ? depk[ra] : 0, ib = (rb < kd) ? depk[rb] : 0;
  double acc_re[4][4], acc_im[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc_re[i][j] = acc_im[i][j] = 0.0;
  for (uint64_t e0 = e_begin; e0 < e_end; e0 += kGK) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int ek = el + 4 * m;
      const uint64_t e = e0 + ek;
      const bool in = e < e_end;
      const uint64_t ie = in ? env_index(dep, e) : 0;
      As[ek][rl] = (in && ra < kd) ? psi[ia | ie] : make_double2(0.0, 0.0);
      Bs[ek][rl] = (in && rb < kd) ? psi[ib | ie] : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kGK; ++kk) {
      double2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // a * conj(b)
          acc_re[i][j] = fma(a[i].x, b[j].x, fma(a[i].y, b[j].y, acc_re[i][j]));
          acc_im[i][j] = fma(a[i].y, b[j].x, fma(-a[i].x, b[j].y, acc_im[i][j]));
        }
    }
    __syncthreads();
  }
  if (part) {
    double2* out = part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (kGT * kGT);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) out[(ty + 16 * i) * kGT + tx + 16 * j] = make_double2(acc_re[i][j], acc_im[i][j]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t r = (uint64_t)tr * kGT + ty + 16 * i, c = (uint64_t)tc * kGT + tx + 16 * j;
      if (r < kd && c < kd && (tr != tc || r <= c)) {
        rho[r * kd + c] = make_double2(acc_re[i][j], r == c ? 0.0 : acc_im[i][j]);
        if (r != c) rho[c * kd + r] = make_double2(acc_re[i][j], -acc_im[i][j]);
      }
    }
}

// sums the nsplit partial tiles in split order and writes rho (both triangles)
__global__ void gram_reduce_kernel(const double2* __restrict__ part, int pairs, int tiles, int nsplit, uint64_t kd,
                                   double2* __restrict__ rho) {
  const uint64_t total = (uint64_t)pairs * kGT * kGT;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const int pair = (int)(t / (kGT * kGT));
    const int w = (int)(t % (kGT * kGT)), rl = w / kGT, cl = w % kGT;
    int tr = 0, rem = pair;
    while (rem >= tiles - tr) {
      rem -= tiles - tr;
      ++tr;
    }
    const int tc = tr + rem;
    const uint64_t r = (uint64_t)tr * kGT + rl, c = (uint64_t)tc * kGT + cl;
    if (r >= kd || c >= kd || (tr == tc && r > c)) continue;
    double re = 0.0, im = 0.0;
    for (int s = 0; s < nsplit; ++s) {
      const double2 v = part[((size_t)s * pairs + pair) * (kGT * kGT) + w];
      re += v.x;
      im += v.y;
    }
    rho[r * kd + c] = make_double2(re, r == c ? 0.0 : im);
    if (r != c) rho[c * kd + r] = make_double2(re, -im);
  }
}

// ---- Householder tridiagonalisation (A Hermitian, row-major, n x n), one launch
//
// Per column the textbook form takes four dependent steps (reflector, A v, w,
// rank-2 update), and as kernels of their own their launches and the sweeps'
// 48 B per entry bound it.  Here one cooperative
// launch keeps every CTA for the whole reduction, with ONE grid-wide barrier
// per column: CTAs hold the reflector vectors and compute them redundantly (in
// the same order, so bit for bit alike) from A's next row and p = A v, which
// their owners publish, and one sweep over a CTA's rows applies the previous
// column's rank-2 update and accumulates the next p.  Up to n = 1024 the rows
// live in shared memory (8 rows per CTA: 128 KiB) and a sweep touches no global
// memory; at 2048 and 4096 they stay in global memory (32 B per entry and
// column), cyclically dealt.  A thread takes one column of 8 (global: 4) rows at
// a time, so the three vectors are read once per 8 rows.  Whole half-cut entropy
// (Gram matrix and eigenvalues included), four launches per column -> this: 14
// qubits (n = 128) 3.9 -> 0.85 ms, 20 (1024) 34.5 -> 8.6, 22 (2048) 89 -> 34,
// 24 (4096) ~400 -> ~220; a column costs ~6 us at n <= 1024: the barrier and the
// chain load - reduce - divide around it.
constexpr uint64_t kHhWaitNs = 2000000000ull;

__device__ __forceinline__ uint64_t clock_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// All CTAs of a cooperative launch; `arrived` counts up for the whole launch.
// Gives up after kHhWaitNs, sets *status and returns false in every CTA.
__device__ bool grid_barrier(unsigned* arrived, unsigned target, int* status, int* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrived, 1u);
    bool ok = true;
    const uint64_t t0 = clock_ns();
    for (;;) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
      if (v >= target) break;
      if (clock_ns() - t0 > kHhWaitNs) {
        atomicExch(status, 1);
        ok = false;
        break;
      }
    }
    *s_ok = ok && *reinterpret_cast<volatile int*>(status) == 0;
  }
  __syncthreads();
  return *s_ok;
}

__device__ __forceinline__ double2 conj_mul(double2 a, double2 b) {   // a conj(b)
  return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -(a.x * b.y)));
}

// sums of x and y over the block in every thread; `red` alternates between calls
__device__ __forceinline__ double2 block_allsum2(double2 v, double2* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double2 t = make_double2(0.0, 0.0);
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) {
    t.x += red[i].x;
    t.y += red[i].y;
  }
  return t;
}

// rowbuf, pbuf: 2 n each (columns alternate); arrived, status: zeroed; n = NT * NPT
template <bool SMEM, int NT, int NPT, int ROWS>
__global__ void __launch_bounds__(NT) hh_fused_kernel(double2* __restrict__ A, int n, double2* rowbuf, double2* pbuf,
                                                      double* __restrict__ d, double* __restrict__ e,
                                                      unsigned* arrived, int* status) {
  extern __shared__ __align__(16) unsigned char hh_smem[];
  double2* vo = reinterpret_cast<double2*>(hh_smem);   // previous reflector
  double2* vn = vo + n;                                // this column's
  double2* const wo = vn + n;                          // previous w
  double2* const rows = wo + n;                        // SMEM: rows blockIdx.x + gridDim.x * r
  __shared__ double2 red[2][NT / 32];
  __shared__ double2 pred[ROWS][NT / 32];
  __shared__ int s_ok;
  const int tid = threadIdx.x, G = gridDim.x, b = blockIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int j = tid; j < n; j += NT) vo[j] = wo[j] = make_double2(0.0, 0.0);
  if (SMEM)
    for (int r = 0; r < ROWS; ++r) {
      const int i = b + G * r;
      if (i < n)
        for (int j = tid; j < n; j += NT) rows[(size_t)r * n + j] = A[(size_t)i * n + j];
    }
  if (b == 0)
    for (int j = tid; j < n; j += NT) rowbuf[j] = A[j];
  if (!grid_barrier(arrived, (unsigned)G, status, &s_ok)) return;
  for (int k = 0; k < n; ++k) {
    const double2* p = pbuf + (size_t)((k + 1) & 1) * n;
    const double2* arow = rowbuf + (size_t)(k & 1) * n;
    const double2 zero = make_double2(0.0, 0.0);
    double2 av[NPT], pv[NPT];          // this thread's entries of row k and of the previous p (columns >= k)
#pragma unroll
    for (int t = 0; t < NPT; ++t) {
      const int j = tid + t * NT;
      pv[t] = (k > 0 && j >= k) ? __ldcg(p + j) : zero;
      av[t] = j >= k ? __ldcg(arow + j) : zero;
    }
    double2 K = zero;                  // v^H p
    if (k > 0) {
#pragma unroll
      for (int t = 0; t < NPT; ++t) {
        const int j = tid + t * NT;
        if (j < k) continue;
        const double2 x = vo[j], y = pv[t];
        K.x += x.x * y.x + x.y * y.y;
        K.y += x.x * y.y - x.y * y.x;
      }
      K = block_allsum2(K, red[0]);
#pragma unroll
      for (int t = 0; t < NPT; ++t) {  // w = 2 (p - K v)
        const int j = tid + t * NT;
        if (j < k) continue;
        const double2 x = vo[j], y = pv[t];
        wo[j] = make_double2(2.0 * (y.x - (K.x * x.x - K.y * x.y)), 2.0 * (y.y - (K.x * x.y + K.y * x.x)));
      }
      __syncthreads();
    }
    // row k with the previous update: a_j = A[k][j] - v_k conj(w_j) - w_k conj(v_j); x_j = conj(a_j)
    const double2 vk = vo[k], wk = wo[k];
    double2 s2 = zero;
#pragma unroll
    for (int t = 0; t < NPT; ++t) {
      const int j = tid + t * NT;
      if (j < k) continue;
      const double2 s = conj_mul(vk, wo[j]), u = conj_mul(wk, vo[j]);
      const double2 a = make_double2(av[t].x - s.x - u.x, av[t].y - s.y - u.y);
      if (j == k) {
        if (b == 0) d[k] = a.x;
        continue;
      }
      av[t] = make_double2(a.x, -a.y);
      if (j == k + 1) vn[j] = av[t];
      s2.x += a.x * a.x + a.y * a.y;
    }
    if (k + 1 == n) return;
    const double xn2 = block_allsum2(s2, red[1]).x;   // its barrier also shows vn[k + 1] to everyone
    // v = (x - alpha e_0) / |x - alpha e_0|, alpha = -phase(x_0) |x|
    const double xn = sqrt(xn2);
    if (b == 0 && tid == 0) e[k] = xn;
    const double2 x0 = vn[k + 1];
    const double ax0 = sqrt(x0.x * x0.x + x0.y * x0.y);
    const double2 ph = ax0 > 0.0 ? make_double2(x0.x / ax0, x0.y / ax0) : make_double2(1.0, 0.0);
    const double2 v0 = make_double2(x0.x + ph.x * xn, x0.y + ph.y * xn);
    const double vn2 = v0.x * v0.x + v0.y * v0.y + (xn2 - (x0.x * x0.x + x0.y * x0.y));
    const double inv = (xn > 0.0 && vn2 > 0.0) ? 1.0 / sqrt(vn2) : 0.0;   // 0: nothing to reflect, v = 0
    __syncthreads();
#pragma unroll
    for (int t = 0; t < NPT; ++t) {
      const int j = tid + t * NT;
      if (j <= k) continue;
      const double2 x = j == k + 1 ? v0 : av[t];
      vn[j] = make_double2(x.x * inv, x.y * inv);
    }
    __syncthreads();
    // this CTA's rows below k: the previous update, then p_i = sum_j A[i][j] v_j
    double2* const pout = pbuf + (size_t)(k & 1) * n;
    double2* const next = rowbuf + (size_t)((k + 1) & 1) * n;
    for (int r0 = 0; b + G * r0 < n; r0 += ROWS) {
      if (b + G * (r0 + ROWS - 1) <= k) continue;   // every row of the group is done
      const int publish = (k + 1 - b) % G == 0 ? (k + 1 - b) / G - r0 : -1;   // the group's row k + 1, if it holds it
      double2* at[ROWS];
      double2 vi[ROWS], wi[ROWS], acc[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int i = b + G * (r0 + r);
        const bool on = i > k && i < n;
        at[r] = on ? (SMEM ? rows + (size_t)r * n : A + (size_t)i * n) : nullptr;
        vi[r] = on ? vo[i] : make_double2(0.0, 0.0);
        wi[r] = on ? wo[i] : make_double2(0.0, 0.0);
        acc[r] = make_double2(0.0, 0.0);
      }
      for (int j = k + 1 + tid; j < n; j += NT) {
        const double2 vj = vo[j], wj = wo[j], u = vn[j];
        double2 a[ROWS];               // all loads before the first store
#pragma unroll
        for (int r = 0; r < ROWS; ++r) a[r] = at[r] ? at[r][j] : zero;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const double2 s = conj_mul(vi[r], wj), t = conj_mul(wi[r], vj);
          a[r].x -= s.x + t.x;
          a[r].y -= s.y + t.y;
          acc[r].x = fma(a[r].x, u.x, fma(-a[r].y, u.y, acc[r].x));
          acc[r].y = fma(a[r].x, u.y, fma(a[r].y, u.x, acc[r].y));
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          if (at[r]) {
            at[r][j] = a[r];
            if (r == publish) __stcg(next + j, a[r]);
          }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          acc[r].x += __shfl_xor_sync(0xffffffffu, acc[r].x, o);
          acc[r].y += __shfl_xor_sync(0xffffffffu, acc[r].y, o);
        }
        if (lane == 0) pred[r][warp] = acc[r];
      }
      __syncthreads();
      if (tid < ROWS) {
        const int i = b + G * (r0 + tid);
        if (i > k && i < n) {
          double2 t = make_double2(0.0, 0.0);
          for (int w = 0; w < NT / 32; ++w) {
            t.x += pred[tid][w].x;
            t.y += pred[tid][w].y;
          }
          __stcg(pout + i, t);
        }
      }
      __syncthreads();
    }
    if (!grid_barrier(arrived, (unsigned)G * (unsigned)(k + 2), status, &s_ok)) return;
    double2* const sw = vo;            // this column's reflector is the next one's previous
    vo = vn;
    vn = sw;
  }
}

// n <= kHhFusedMax, n a power of two >= 128
cudaError_t launch_hh_fused(double2* A, int n, double2* rowbuf, double2* pbuf, double* d, double* e, unsigned* arrived,
                            int* status, cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (const char* v = getenv("IQ_ENTROPY_SMS")) sms = std::max(1, std::min(sms, atoi(v)));
  const HhShape h = hh_shape(n, sms);
  const void* fn = nullptr;
  auto use = [&](const void* f, bool smem_rows, int threads, int rows) {
    if (h.smem_rows == smem_rows && h.threads == threads && h.rows == rows) fn = f;
  };
  constexpr int RS = kHhRows, RG = kHhRows / 2;
  switch (n) {
    case 128:
      use((const void*)hh_fused_kernel<true, 128, 1, RS>, true, 128, RS);
      use((const void*)hh_fused_kernel<false, 128, 1, RG>, false, 128, RG);
      break;
    case 256:
      use((const void*)hh_fused_kernel<true, 256, 1, RS>, true, 256, RS);
      use((const void*)hh_fused_kernel<false, 256, 1, RG>, false, 256, RG);
      break;
    case 512:
      use((const void*)hh_fused_kernel<true, 256, 2, RS>, true, 256, RS);
      use((const void*)hh_fused_kernel<false, 512, 1, RG>, false, 512, RG);
      break;
    case 1024:
      use((const void*)hh_fused_kernel<true, 256, 4, RS>, true, 256, RS);
      use((const void*)hh_fused_kernel<false, 512, 2, RG>, false, 512, RG);
      break;
    case 2048: use((const void*)hh_fused_kernel<false, 512, 4, RG>, false, 512, RG); break;
    case 4096: use((const void*)hh_fused_kernel<false, 512, 8, RG>, false, 512, RG); break;
  }
  if (!fn) return cudaErrorInvalidValue;
  cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)h.smem);
  if (err != cudaSuccess) return err;
  void* args[] = {&A, &n, &rowbuf, &pbuf, &d, &e, &arrived, &status};
  return cudaLaunchCooperativeKernel(fn, dim3(h.grid), dim3(h.threads), args, h.smem, st);
}

// ---- the same column by column, for n above kHhFusedMax (sweeps of 1 GiB dwarf their launches)

// Reflector for column k: x_j = A[j][k] = conj(A[k][j]) for j > k.
// v = (x - alpha e_{k+1}) / |x - alpha e_{k+1}|, alpha = -phase(x_{k+1}) |x|.
// Writes v[j] (j > k), d[k] = Re A[k][k], e[k] = |alpha|, flag = 0 when x = 0.
__global__ void hh_vector_kernel(const double2* __restrict__ A, int n, int k, double2* __restrict__ v,
                                 double* __restrict__ d, double* __restrict__ e, int* __restrict__ flag) {
  __shared__ double red[32];
  const size_t row = (size_t)k * n;
  double s = 0.0;
  for (int j = k + 1 + threadIdx.x; j < n; j += blockDim.x) {
    const double2 a = A[row + j];
    s += a.x * a.x + a.y * a.y;
  }
  const double xn2 = block_allsum(s, red);
  const double xn = sqrt(xn2);
  const double2 a0 = A[row + k + 1];
  const double2 x0 = make_double2(a0.x, -a0.y);
  const double ax0 = hypot(x0.x, x0.y);
  const double2 ph = ax0 > 0.0 ? make_double2(x0.x / ax0, x0.y / ax0) : make_double2(1.0, 0.0);
  const double2 alpha = make_double2(-ph.x * xn, -ph.y * xn);
  const double2 v0 = make_double2(x0.x - alpha.x, x0.y - alpha.y);
  // |v|^2 = |x0 - alpha|^2 + (|x|^2 - |x0|^2)
  const double vn2 = v0.x * v0.x + v0.y * v0.y + (xn2 - (x0.x * x0.x + x0.y * x0.y));
  const bool ok = xn > 0.0 && vn2 > 0.0;
  const double inv = ok ? 1.0 / sqrt(vn2) : 0.0;
  for (int j = k + 1 + threadIdx.x; j < n; j += blockDim.x) {
    double2 x;
    if (j == k + 1) {
      x = v0;
    } else {
      const double2 a = A[row + j];
      x = make_double2(a.x, -a.y);
    }
    v[j] = make_double2(x.x * inv, x.y * inv);
  }
  if (threadIdx.x == 0) {
    d[k] = A[row + k].x;
    e[k] = xn;
    *flag = ok ? 1 : 0;
  }
}

// p_i = sum_{j > k} A[i][j] v_j for i > k; one warp per row
__global__ void hh_hemv_kernel(const double2* __restrict__ A, int n, int k, const double2* __restrict__ v,
                               const int* __restrict__ flag, double2* __restrict__ p) {
  if (!*flag) return;
  const int lane = threadIdx.x & 31;
  const int i = k + 1 + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const double2* row = A + (size_t)i * n;
  double re = 0.0, im = 0.0;
  for (int j = k + 1 + lane; j < n; j += 32) {
    const double2 a = row[j], b = v[j];
    re = fma(a.x, b.x, fma(-a.y, b.y, re));
    im = fma(a.x, b.y, fma(a.y, b.x, im));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
  }
  if (lane == 0) p[i] = make_double2(re, im);
}

// K = v^H p, w = 2 (p - K v)
__global__ void hh_w_kernel(int n, int k, const double2* __restrict__ v, const double2* __restrict__ p,
                            const int* __restrict__ flag, double2* __restrict__ w) {
  if (!*flag) return;
  __shared__ double red[32];
  double kr = 0.0, ki = 0.0;
  for (int j = k + 1 + threadIdx.x; j < n; j += blockDim.x) {
    const double2 a = v[j], b = p[j];
    // conj(a) * b
    kr += a.x * b.x + a.y * b.y;
    ki += a.x * b.y - a.y * b.x;
  }
  kr = block_allsum(kr, red);
  __syncthreads();
  ki = block_allsum(ki, red);
  for (int j = k + 1 + threadIdx.x; j < n; j += blockDim.x) {
    const double2 a = v[j], b = p[j];
    w[j] = make_double2(2.0 * (b.x - (kr * a.x - ki * a.y)), 2.0 * (b.y - (kr * a.y + ki * a.x)));
  }
}

// A[i][j] -= v_i conj(w_j) + w_i conj(v_j) for i, j > k
__global__ void hh_her2_kernel(double2* __restrict__ A, int n, int k, const double2* __restrict__ v,
                               const double2* __restrict__ w, const int* __restrict__ flag) {
  if (!*flag) return;
  const int j = k + 1 + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double2 vj = v[j], wj = w[j];
  for (int i = k + 1 + blockIdx.y; i < n; i += gridDim.y) {
    const double2 vi = v[i], wi = w[i];
    double2 a = A[(size_t)i * n + j];
    // v_i conj(w_j) + w_i conj(v_j)
    const double re = vi.x * wj.x + vi.y * wj.y + wi.x * vj.x + wi.y * vj.y;
    const double im = vi.y * wj.x - vi.x * wj.y + wi.y * vj.x - wi.x * vj.y;
    a.x -= re;
    a.y -= im;
    A[(size_t)i * n + j] = a;
  }
}

// the last 2 x 2 block
__global__ void hh_tail_kernel(const double2* __restrict__ A, int n, double* __restrict__ d, double* __restrict__ e) {
  if (threadIdx.x != 0) return;
  if (n >= 2) {
    d[n - 2] = A[(size_t)(n - 2) * n + n - 2].x;
    const double2 b = A[(size_t)(n - 1) * n + n - 2];
    e[n - 2] = hypot(b.x, b.y);
  }
  d[n - 1] = A[(size_t)(n - 1) * n + n - 1].x;
}

// number of eigenvalues of the tridiagonal (d, squares e2) below x (Sturm count)
__device__ int sturm_count(const double* __restrict__ d, const double* __restrict__ e2, int n, double x,
                           double pivmin) {
  int cnt = 0;
  double q = d[0] - x;
  if (fabs(q) < pivmin) q = -pivmin;
  if (q < 0.0) ++cnt;
  for (int i = 1; i < n; ++i) {
    q = (d[i] - x) - e2[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    if (q < 0.0) ++cnt;
  }
  return cnt;
}

// e <- e^2 and the Gershgorin interval: bounds[0] = lo, [1] = hi, [2] = pivmin (one CTA)
__global__ void __launch_bounds__(256) gershgorin_kernel(const double* __restrict__ d, double* __restrict__ e, int n,
                                                         double* __restrict__ bounds) {
  __shared__ double slo[256], shi[256], sm[256];
  const int tid = threadIdx.x;
  double lo = d[0], hi = d[0], emax2 = 0.0;
  for (int t = tid; t < n; t += 256) {
    const double r = (t > 0 ? e[t - 1] : 0.0) + (t + 1 < n ? e[t] : 0.0);
    lo = fmin(lo, d[t] - r);
    hi = fmax(hi, d[t] + r);
    if (t + 1 < n) emax2 = fmax(emax2, e[t] * e[t]);
  }
  slo[tid] = lo;
  shi[tid] = hi;
  sm[tid] = emax2;
  __syncthreads();
  for (int t = tid; t + 1 < n; t += 256) e[t] = e[t] * e[t];
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o) {
      slo[tid] = fmin(slo[tid], slo[tid + o]);
      shi[tid] = fmax(shi[tid], shi[tid + o]);
      sm[tid] = fmax(sm[tid], sm[tid + o]);
    }
    __syncthreads();
  }
  if (tid == 0) {
    const double span = fmax(fabs(slo[0]), fabs(shi[0]));
    bounds[0] = slo[0] - (2.0 * DBL_EPSILON * span * n + 1e-300);
    bounds[1] = shi[0] + (2.0 * DBL_EPSILON * span * n + 1e-300);
    bounds[2] = 1e-290 * fmax(1.0, sm[0]);
  }
}

// eig[i] = i-th smallest eigenvalue, one warp each: 32 Sturm counts split the
// interval into 33 per step (a count is a serial chain of n divisions, so one
// thread's bisection took 52 of them; this takes 11 side by side)
__global__ void bisect_kernel(const double* __restrict__ d, const double* __restrict__ e2, int n,
                              const double* __restrict__ bounds, double* __restrict__ eig) {
  const int lane = threadIdx.x & 31;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  double lo = bounds[0], hi = bounds[1];
  const double pivmin = bounds[2];
  for (int it = 0; it < 256; ++it) {
    if (hi - lo <= 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + 1e-300) break;
    const double h = (hi - lo) / 33.0;
    const double x = fma((double)(lane + 1), h, lo);
    const bool above = sturm_count(d, e2, n, x, pivmin) > i;   // the eigenvalue lies below x
    const unsigned m = __ballot_sync(0xffffffffu, above);
    const int first = m ? __ffs(m) - 1 : 32;                   // lowest point above the eigenvalue
    const double nlo = first > 0 ? __shfl_sync(0xffffffffu, x, first - 1) : lo;
    const double nhi = first < 32 ? __shfl_sync(0xffffffffu, x, first & 31) : hi;
    if (!(nlo > lo || nhi < hi)) break;                        // the interval is one rounding wide
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) eig[i] = 0.5 * (lo + hi);
}

uint64_t deposit(uint64_t x, const int* bits, int nb) {
  uint64_t r = 0;
  for (int b = 0; b < nb; ++b)
    if ((x >> b) & 1) r |= 1ULL << bits[b];
  return r;
}

}  // namespace

int reduced_spectrum_max_bits() { return 13; }

namespace {

struct SpectrumLayout {
  int tiles, pairs, nsplit;
  size_t rho, part, vec, small, dep, total;   // byte offsets and the whole
};

SpectrumLayout spectrum_layout(int nbits, int k) {
  SpectrumLayout L;
  const int nt = nbits - k;
  const size_t n = (size_t)1 << k;
  const uint64_t ed = 1ULL << nt;
  L.tiles = (int)((n + kGT - 1) / kGT);
  L.pairs = L.tiles * (L.tiles + 1) / 2;
  // split the environment so that at least ~4 CTAs per SM run, in chunks of >= 256 entries
  L.nsplit = 1;
  while ((uint64_t)L.pairs * L.nsplit < 4 * 148 && ed / (2ULL * L.nsplit) >= 256) L.nsplit *= 2;
  auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
  size_t off = 0;
  L.rho = off;
  off = align(off + n * n * sizeof(double2));
  L.part = off;
  if (L.nsplit > 1) off = align(off + (size_t)L.nsplit * L.pairs * kGT * kGT * sizeof(double2));
  L.vec = off;
  off = align(off + 4 * n * sizeof(double2) + 3 * n * sizeof(double));
  L.small = off;
  off = align(off + 256);
  L.dep = off;
  const int lobits = (nt + 1) / 2;
  off = align(off + (n + (1ULL << lobits) + (1ULL << (nt - lobits))) * sizeof(uint64_t));
  L.total = off;
  return L;
}

}  // namespace

size_t reduced_spectrum_bytes(int nbits, int k) { return spectrum_layout(nbits, k).total; }

cudaError_t reduced_spectrum(const double2* psi, int nbits, const int* keep, int k, std::vector<double>& eig, void* work,
                             cudaStream_t st) {
  if (k < 7 || k > reduced_spectrum_max_bits() || k >= nbits || !work) return cudaErrorInvalidValue;
  std::vector<int> traced;
  for (int q = 0; q < nbits; ++q) {
    bool in = false;
    for (int i = 0; i < k; ++i) in |= keep[i] == q;
    if (!in) traced.push_back(q);
  }
  const int nt = (int)traced.size();
  const uint64_t kd = 1ULL << k, ed = 1ULL << nt;
  const int lobits = (nt + 1) / 2, hibits = nt - lobits;
  std::vector<uint64_t> h_depk(kd), h_lo(1ULL << lobits), h_hi(1ULL << hibits);
  for (uint64_t r = 0; r < kd; ++r) h_depk[r] = deposit(r, keep, k);
  for (uint64_t x = 0; x < h_lo.size(); ++x) h_lo[x] = deposit(x, traced.data(), lobits);
  for (uint64_t x = 0; x < h_hi.size(); ++x) h_hi[x] = deposit(x, traced.data() + lobits, hibits);

  const SpectrumLayout L = spectrum_layout(nbits, k);
  const int tiles = L.tiles, pairs = L.pairs, nsplit = L.nsplit;
  const uint64_t per = ed / nsplit;
  const size_t n = (size_t)kd;
  char* const buf = static_cast<char*>(work);
  double2* rho = reinterpret_cast<double2*>(buf + L.rho);
  double2* part = nsplit > 1 ? reinterpret_cast<double2*>(buf + L.part) : nullptr;
  double2* v = reinterpret_cast<double2*>(buf + L.vec);   // 4 n: row and p buffers, or v, p, w
  double* d = reinterpret_cast<double*>(v + 4 * n);
  double* e = d + n;
  double* ev = e + n;
  int* flag = reinterpret_cast<int*>(buf + L.small);      // [0] flag / status, [1] barrier count, then 3 doubles
  double* bounds = reinterpret_cast<double*>(buf + L.small + 64);
  uint64_t* depk = reinterpret_cast<uint64_t*>(buf + L.dep);
  uint64_t* lo = depk + h_depk.size();
  uint64_t* hi = lo + h_lo.size();

  cudaError_t err = cudaMemsetAsync(flag, 0, 64, st);
  if (err == cudaSuccess) err = cudaMemcpyAsync(depk, h_depk.data(), h_depk.size() * 8, cudaMemcpyHostToDevice, st);
  if (err == cudaSuccess) err = cudaMemcpyAsync(lo, h_lo.data(), h_lo.size() * 8, cudaMemcpyHostToDevice, st);
  if (err == cudaSuccess) err = cudaMemcpyAsync(hi, h_hi.data(), h_hi.size() * 8, cudaMemcpyHostToDevice, st);
  uint64_t launches = 0;
  if (err == cudaSuccess) {
    EnvDep dep{lo, hi, lobits};
    gram_kernel<<<dim3(pairs, nsplit), kGThreads, 0, st>>>(psi, depk, dep, tiles, kd, per, part, rho);
    ++launches;
    if (nsplit > 1) {
      gram_reduce_kernel<<<std::min<uint64_t>(((uint64_t)pairs * kGT * kGT + 255) / 256, 148 * 16), 256, 0, st>>>(
          part, pairs, tiles, nsplit, kd, rho);
      ++launches;
    }
    err = cudaGetLastError();
  }
  const int nn = (int)n;
  if (err == cudaSuccess && nn <= kHhFusedMax) {
    err = launch_hh_fused(rho, nn, v, v + 2 * n, d, e, reinterpret_cast<unsigned*>(flag + 1), flag, st);
    ++launches;
  } else {
    double2 *p = v + n, *w = p + n;
    for (int kcol = 0; err == cudaSuccess && kcol + 2 < nn; ++kcol) {
      const int m = nn - kcol - 1;
      hh_vector_kernel<<<1, 1024, 0, st>>>(rho, nn, kcol, v, d, e, flag);
      hh_hemv_kernel<<<(m + 7) / 8, 256, 0, st>>>(rho, nn, kcol, v, flag, p);
      hh_w_kernel<<<1, 1024, 0, st>>>(nn, kcol, v, p, flag, w);
      const int gy = std::min(m, 256);
      hh_her2_kernel<<<dim3((m + 127) / 128, gy), 128, 0, st>>>(rho, nn, kcol, v, w, flag);
      launches += 4;
      err = cudaGetLastError();
    }
    if (err == cudaSuccess) {
      hh_tail_kernel<<<1, 32, 0, st>>>(rho, nn, d, e);
      cudaMemsetAsync(flag, 0, sizeof(int), st);   // the status read below
      ++launches;
    }
  }
  if (err == cudaSuccess) {
    gershgorin_kernel<<<1, 256, 0, st>>>(d, e, nn, bounds);
    bisect_kernel<<<(nn + 3) / 4, 128, 0, st>>>(d, e, nn, bounds, ev);
    launches += 2;
    err = cudaGetLastError();
  }
  count_launches(launches);
  eig.assign(n, 0.0);
  if (err == cudaSuccess) err = cudaMemcpyAsync(eig.data(), ev, n * sizeof(double), cudaMemcpyDeviceToHost, st);
  int status = 0;
  if (err == cudaSuccess) err = cudaMemcpyAsync(&status, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
  const cudaError_t serr = cudaStreamSynchronize(st);
  if (err == cudaSuccess) err = serr;
  if (err == cudaSuccess && status != 0) err = cudaErrorLaunchTimeout;   // a grid barrier gave up
  return err;
}

}  // namespace iqb
