// iq_resident.cu -- persistent executor for the small circuits of a gradient
// batch.
//
// A circuit of n <= kResidentMaxQubits qubits keeps psi and lambda (2 x 16 B x
// 2^n, 128 KiB at 12 qubits) in one CTA's shared memory for its whole adjoint
// gradient: forward, lambda = H psi, then the backward sweep (per rotation: the
// term Im<lambda|P|psi> and the inverse rotation on both vectors), with no
// global-memory traffic but the parameters in and the energy and gradient out.
// All (circuit, parameter set) items of a batch are the entries of a
// device-side queue, largest first; one persistent launch of as many CTAs as
// fit the GPU pops them with an atomic counter until the queue is empty (no CTA
// ever waits for another).  The launch, with the parameter upload before it and
// the result download after it, is captured once per batch structure as a CUDA
// graph and replayed.
//
// The gates run in stages (schedule() below): each thread holds the 2^K
// amplitudes of both vectors that K index bits span and applies every gate of
// the stage whose target is one of those bits, so a stage costs one round trip
// through shared memory and one barrier, not one of each per gate.  What bounds
// a small circuit is the chain of dependent steps, so nothing but the gates
// stays on it: a stage's steps and the sines and cosines of its angles are
// fetched by the last warp during the stage before, and the gradient terms of
// up to four rotations are summed over a warp at once, over the CTA's warps
// after the barrier that ends the stage.
//
// Rotations are exp(-i t P / 2); U3 = e^{i(phi+lambda)/2} Rz(phi) Ry(theta)
// Rz(lambda) with the global phase dropped, P(l) as Rz(l) (the energy does not
// see a global phase) -- the conventions of the tile-pass executor
// (ansatz_forward / ansatz_backward in iq_sched.cpp).  The gradient term and
// the inverse rotation are the expressions the tile kernels use
// (grad_term / unrotate in iq_pipe.cuh).  Each item is computed by one CTA in
// a fixed order: results are reproducible bit for bit.
#include "iq_resident.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <type_traits>
#include <map>
#include <memory>
#include <mutex>

#include "iq_pipe.cuh"

namespace iqb {
namespace {

constexpr int kResThreads = 256;
constexpr int kResWarps = kResThreads / 32;
constexpr int kStageSteps = 32;   // steps of a stage: one lane of the fetching warp each
constexpr int kStageRots = 16;    // rotations of a stage, no two of one parameter
constexpr int kRing = 4;          // rotations whose terms a warp sums at once
constexpr int kRingRow = 40;      // doubles per ring row: two rows (a half-warp's loads) on different banks
constexpr int kWideStageBits = 11;   // index bits from which a stage has three bits (stage_bits)
constexpr int kMinBits = 3;       // circuits of fewer qubits run as three, the others idle in |0>

enum ResKind { RES_RX = 0, RES_RY, RES_RZ, RES_H, RES_X, RES_SX, RES_CX, RES_CZ };

// one step of a stage: x = kind * 4 + position of its target among the stage's
// bits (-1: no step); rotations: y = parameter, z = number among the stage's
// rotations; CX, CZ: y = mask of the other bits that have to be set, z = the
// thread's amplitudes (bit i for amplitude i) for which its own bits allow it
using ResStep = int4;

struct ResCirc {
  int n, nst, st0, nparams;   // index bits (>= kMinBits); stages and the first of them
  int ngroups, g0, t0, k;     // k: bits of a stage
  uint64_t param0;   // first parameter of set 0 in the parameter array
  uint64_t e0;       // first energy slot
  uint64_t grad0;    // first gradient slot (set-major, nparams per set)
};

// position of amplitude x in shared memory: the 16-byte bank group takes the
// next three bits too, so stages on bits 0-2 and on higher bits are both free
// of bank conflicts (linear: sw(x ^ y) = sw(x) ^ sw(y))
__device__ __forceinline__ uint32_t sw(uint32_t x) { return x ^ ((x >> 3) & 7u); }

__device__ __forceinline__ uint32_t insert0(uint32_t p, int q) {
  const uint32_t lo = p & ((1u << q) - 1u);
  return ((p >> q) << (q + 1)) | lo;
}

// forward (sign = -1) or inverse (sign = +1) rotation exp(-/+ i t P / 2) on one
// pair, as the structured matrix unrotate() takes
template <int GEN>
__device__ __forceinline__ void rot_pair(double c, double s, double2& x0, double2& x1) {
  double2 y0, y1;
  if (GEN == 2) unrotate<2>(x0, x1, y0, y1, make_double2(c, s), make_double2(0.0, 0.0), make_double2(c, -s));
  else if (GEN == 1) unrotate<1>(x0, x1, y0, y1, make_double2(c, 0.0), make_double2(s, 0.0), make_double2(c, 0.0));
  else unrotate<0>(x0, x1, y0, y1, make_double2(c, 0.0), make_double2(0.0, s), make_double2(c, 0.0));
  x0 = y0;
  x1 = y1;
}

// a fixed one-qubit gate (or its inverse) on one pair
template <int KIND, bool INVERSE>
__device__ __forceinline__ void fixed1_pair(double2& x0, double2& x1) {
  if (KIND == RES_H) {
    const double r = 0.70710678118654752440;
    const double2 a = x0, b = x1;
    x0 = make_double2(r * (a.x + b.x), r * (a.y + b.y));
    x1 = make_double2(r * (a.x - b.x), r * (a.y - b.y));
  } else if (KIND == RES_X) {
    const double2 t = x0;
    x0 = x1;
    x1 = t;
  } else {   // SX = 1/2 [[1+i, 1-i], [1-i, 1+i]]; its inverse is the conjugate
    const double sg = INVERSE ? -1.0 : 1.0;
    const double2 a = x0, b = x1;
    // (1 + i sg) a / 2 + (1 - i sg) b / 2 and the mirror
    x0 = make_double2(0.5 * (a.x - sg * a.y + b.x + sg * b.y), 0.5 * (a.y + sg * a.x + b.y - sg * b.x));
    x1 = make_double2(0.5 * (a.x + sg * a.y + b.x - sg * b.y), 0.5 * (a.y - sg * a.x + b.y + sg * b.x));
  }
}

// block sum in a fixed order (warps by shuffles, then the warp sums in order); valid in thread 0
__device__ __forceinline__ double block_sum_fixed(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kResThreads / 32; ++w) t += red[w];
  __syncthreads();
  return t;
}

// what a stage's threads share: steps and angles of the stage at hand and of the
// next one, the warps' sums of its gradient terms
struct ResShared {
  ResStep steps[2][kStageSteps];
  double2 cs[2][kStageRots];   // cos, sin of half the angle
  int4 head[2];                // x: steps, y: rotations, z: the bits (8 bits each)
  double wsum[2][kStageRots][kResWarps];
  double ring[kResWarps][kRing * kRingRow];
  double red[kResWarps];
  int item;
};

// the fetching warp brings stage st into buffer b
__device__ __forceinline__ void fetch_stage(ResShared& S, int b, const int4* __restrict__ heads,
                                            const ResStep* __restrict__ steps, int st, const double* th) {
  const int lane = threadIdx.x & 31;
  const ResStep s = steps[(size_t)st * kStageSteps + lane];
  if (lane == 0) S.head[b] = heads[st];
  S.steps[b][lane] = s;
  if (s.x >= 0 && (s.x >> 2) <= RES_RZ) {
    double sn, c;
    sincos(0.5 * th[s.y], &sn, &c);
    S.cs[b][s.z] = make_double2(c, sn);
  }
}

// amplitude pairs of local bit J
template <int K, int J, class F>
__device__ __forceinline__ void each_pair(F f) {
#pragma unroll
  for (int p = 0; p < (1 << (K - 1)); ++p) {
    const int i0 = ((p >> J) << (J + 1)) | (p & ((1 << J) - 1));
    f(i0, i0 | (1 << J));
  }
}

// sums of the warp's last `cnt` rows of the ring: rows hold rotations hi, hi - 1, ...
__device__ __forceinline__ void flush_ring(ResShared& S, int b, int hi, int cnt, bool add) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, row = lane >> 3;
  __syncwarp();
  const double* r = S.ring[w] + row * kRingRow + (lane & 7);
  double v = row < cnt ? (r[0] + r[8]) + (r[16] + r[24]) : 0.0;
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  if ((lane & 7) == 0 && row < cnt) {
    double& t = S.wsum[b][hi - row][w];
    t = add ? t + v : v;
  }
  __syncwarp();
}

// One step on a thread's amplitudes; BACK: the inverse, on both vectors, and a
// rotation's gradient term into `acc`.
template <int K, int J, bool BACK>
__device__ __forceinline__ void step_on_bit(int kind, const ResStep& s, const double2* cs, uint32_t base,
                                            double2 (&a)[1 << K], double2 (&l)[1 << K], double& acc) {
  if (kind <= RES_RZ) {
    const double2 t = cs[s.z];
    const double c = t.x, sn = BACK ? t.y : -t.y;
    auto rot = [&](auto gen) {
      constexpr int GEN = decltype(gen)::value;
      each_pair<K, J>([&](int i0, int i1) {
        if (BACK) {
          acc += grad_term<GEN>(a[i0], a[i1], l[i0], l[i1]);
          rot_pair<GEN>(c, sn, l[i0], l[i1]);
        }
        rot_pair<GEN>(c, sn, a[i0], a[i1]);
      });
    };
    if (kind == RES_RX) rot(std::integral_constant<int, 0>{});
    else if (kind == RES_RY) rot(std::integral_constant<int, 1>{});
    else rot(std::integral_constant<int, 2>{});
  } else if (kind == RES_CX) {
    const uint32_t on = (base & (uint32_t)s.y) == (uint32_t)s.y ? (uint32_t)s.z : 0u;
    each_pair<K, J>([&](int i0, int i1) {
      const bool swap = (on >> i0) & 1u;
      const double2 x = a[i0], y = a[i1];
      a[i0] = swap ? y : x;
      a[i1] = swap ? x : y;
      if (BACK) {
        const double2 u = l[i0], v = l[i1];
        l[i0] = swap ? v : u;
        l[i1] = swap ? u : v;
      }
    });
  } else {
    auto fix = [&](auto gate) {
      constexpr int KIND = decltype(gate)::value;
      each_pair<K, J>([&](int i0, int i1) {
        fixed1_pair<KIND, BACK>(a[i0], a[i1]);
        if (BACK) fixed1_pair<KIND, BACK>(l[i0], l[i1]);
      });
    };
    if (kind == RES_H) fix(std::integral_constant<int, RES_H>{});
    else if (kind == RES_X) fix(std::integral_constant<int, RES_X>{});
    else fix(std::integral_constant<int, RES_SX>{});
  }
}

// The stage in buffer b on the whole state: forward on psi, or (BACK) its
// inverse on psi and lambda, with the gradient terms into S.wsum[b].
template <int K, bool BACK>
__device__ __forceinline__ void run_stage(ResShared& S, int b, double2* psi, double2* lam, uint32_t groups) {
  constexpr int A = 1 << K;
  const int4 h = S.head[b];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t off[A];
#pragma unroll
  for (int i = 0; i < A; ++i) {
    uint32_t o = 0;
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (i >> j & 1) o |= 1u << ((h.z >> (8 * j)) & 255);
    off[i] = sw(o);
  }
  // whole warps take part (the ring's sums): lanes past the last group hold zeros
  for (uint32_t g0 = w * 32; g0 < groups; g0 += kResThreads) {
    const bool on = g0 + lane < groups;
    uint32_t base = on ? g0 + lane : 0u;
#pragma unroll
    for (int j = 0; j < K; ++j) base = insert0(base, (h.z >> (8 * j)) & 255);
    const uint32_t at = sw(base);
    double2 a[A], l[A];
#pragma unroll
    for (int i = 0; i < A; ++i) {
      a[i] = on ? psi[at ^ off[i]] : make_double2(0.0, 0.0);
      if (BACK) l[i] = on ? lam[at ^ off[i]] : make_double2(0.0, 0.0);
    }
    int nr = 0;   // rotations so far
    for (int q = 0; q < h.x; ++q) {
      const ResStep s = S.steps[b][BACK ? h.x - 1 - q : q];
      const int kind = s.x >> 2, j = s.x & 3;
      if (kind == RES_CZ) {
        const uint32_t neg = (base & (uint32_t)s.y) == (uint32_t)s.y ? (uint32_t)s.z : 0u;
#pragma unroll
        for (int i = 0; i < A; ++i)
          if ((neg >> i) & 1u) {
            a[i] = make_double2(-a[i].x, -a[i].y);
            if (BACK) l[i] = make_double2(-l[i].x, -l[i].y);
          }
        continue;
      }
      double acc = 0.0;
      if (j == 0) step_on_bit<K, 0, BACK>(kind, s, S.cs[b], base, a, l, acc);
      else if (K == 2 || j == 1) step_on_bit<K, 1, BACK>(kind, s, S.cs[b], base, a, l, acc);
      else step_on_bit<K, K - 1, BACK>(kind, s, S.cs[b], base, a, l, acc);
      if (BACK && kind <= RES_RZ) {
        S.ring[w][(nr & (kRing - 1)) * kRingRow + lane] = acc;
        ++nr;
        if ((nr & (kRing - 1)) == 0) flush_ring(S, b, h.y - 1 - (nr - kRing), kRing, g0 >= kResThreads);
      }
    }
    if (BACK && (nr & (kRing - 1)))
      flush_ring(S, b, h.y - 1 - (nr & ~(kRing - 1)), nr & (kRing - 1), g0 >= kResThreads);
#pragma unroll
    for (int i = 0; i < A; ++i)
      if (on) {
        psi[at ^ off[i]] = a[i];
        if (BACK) lam[at ^ off[i]] = l[i];
      }
  }
}

__global__ void __launch_bounds__(kResThreads, 2) resident_adjoint_kernel(
    const ResCirc* __restrict__ circs, const int2* __restrict__ items, int nitems, int* __restrict__ head,
    const int4* __restrict__ heads, const ResStep* __restrict__ steps, const uint64_t* __restrict__ gx,
    const int* __restrict__ gfirst, const uint64_t* __restrict__ tz, const double2* __restrict__ tc,
    const double* __restrict__ params, double* __restrict__ e_out, double* __restrict__ g_out, int dim_max,
    int params_max) {
  extern __shared__ __align__(16) unsigned char res_smem[];
  double2* const psi = reinterpret_cast<double2*>(res_smem);
  double* const grads = reinterpret_cast<double*>(psi + 2 * (size_t)dim_max);
  double* const th = grads + params_max;
  __shared__ __align__(16) ResShared S;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  for (;;) {
    if (tid == 0) S.item = atomicAdd(head, 1);
    __syncthreads();
    const int it = S.item;
    __syncthreads();
    if (it >= nitems) return;
    const int2 iw = items[it];
    const ResCirc C = circs[iw.x];
    const uint32_t dim = 1u << C.n, groups = dim >> C.k;
    const int warps = (int)((min(groups, (uint32_t)kResThreads) + 31) / 32);   // with a group
    double2* const lam = psi + dim;
    const double* set = params + C.param0 + (uint64_t)iw.y * C.nparams;
    for (uint32_t x = tid; x < dim; x += kResThreads) psi[x] = make_double2(x == 0 ? 1.0 : 0.0, 0.0);
    for (int p = tid; p < C.nparams; p += kResThreads) {
      grads[p] = 0.0;
      th[p] = set[p];
    }
    __syncthreads();
    if (w == kResWarps - 1 && C.nst) fetch_stage(S, 0, heads, steps, C.st0, th);
    __syncthreads();
    // forward
    for (int u = 0; u < C.nst; ++u) {
      if (w == kResWarps - 1) fetch_stage(S, (u + 1) & 1, heads, steps, C.st0 + min(u + 1, C.nst - 1), th);
      if (C.k == 2) run_stage<2, false>(S, u & 1, psi, lam, groups);
      else run_stage<3, false>(S, u & 1, psi, lam, groups);
      __syncthreads();
    }
    // lambda = H psi and the energy
    double e = 0.0;
    for (uint32_t x = tid; x < dim; x += kResThreads) {
      const double2 px = psi[sw(x)];
      double2 l = make_double2(0.0, 0.0);
      for (int g = 0; g < C.ngroups; ++g) {
        const uint64_t xm = gx[C.g0 + g];
        const uint32_t src = x ^ (uint32_t)xm;
        const double2 a = psi[sw(src)];
        double2 f = make_double2(0.0, 0.0);
        for (int t = gfirst[C.g0 + g]; t < gfirst[C.g0 + g + 1]; ++t) {
          const double2 cf = tc[C.t0 + t];
          if (__popcll((uint64_t)src & tz[C.t0 + t]) & 1) { f.x -= cf.x; f.y -= cf.y; }
          else { f.x += cf.x; f.y += cf.y; }
        }
        l = cfma(l, f, a);
      }
      lam[sw(x)] = l;
      e += px.x * l.x + px.y * l.y;
    }
    e = block_sum_fixed(e, S.red);   // ends with a barrier: lambda complete
    if (tid == 0) e_out[C.e0 + iw.y] = e;
    // backward: the stages in reverse, their steps too
    for (int u = C.nst; u < 2 * C.nst; ++u) {
      const int b = u & 1;
      if (w == kResWarps - 1 && u + 1 < 2 * C.nst)
        fetch_stage(S, b ^ 1, heads, steps, C.st0 + 2 * C.nst - 2 - u, th);
      // the summing warp's lane of a step keeps what it needs past the barrier,
      // when the step's buffer may be overwritten
      ResStep mine = make_int4(-1, 0, 0, 0);
      if (w == kResWarps - 2 && lane < S.head[b].x) mine = S.steps[b][lane];
      if (C.k == 2) run_stage<2, true>(S, b, psi, lam, groups);
      else run_stage<3, true>(S, b, psi, lam, groups);
      __syncthreads();
      if (mine.x >= 0 && (mine.x >> 2) <= RES_RZ) {
        double t = 0.0;
        for (int v = 0; v < warps; ++v) t += S.wsum[b][mine.z][v];
        grads[mine.y] += t;
      }
    }
    __syncthreads();
    double* const out = g_out + C.grad0 + (uint64_t)iw.y * C.nparams;
    for (int p = tid; p < C.nparams; p += kResThreads) out[p] = grads[p];
    __syncthreads();
  }
}

size_t smem_bytes(int nmax, int pmax) { return 2 * (sizeof(double2) << nmax) + 2 * (size_t)pmax * sizeof(double); }

// one batch structure: device arrays, pinned staging and the captured graph
struct Plan {
  int dev = -1;
  cudaStream_t stream = nullptr;
  cudaGraphExec_t exec = nullptr;
  size_t nparams_total = 0, nenergies = 0, ngrads = 0;
  std::vector<void*> dbufs;
  double* h_params = nullptr;
  double* h_e = nullptr;
  double* h_g = nullptr;
  ~Plan() {
    if (stream) cudaStreamSynchronize(stream);
    if (exec) cudaGraphExecDestroy(exec);
    for (void* p : dbufs) cudaFree(p);
    if (h_params) cudaFreeHost(h_params);
    if (h_e) cudaFreeHost(h_e);
    if (h_g) cudaFreeHost(h_g);
    if (stream) cudaStreamDestroy(stream);
  }
};

uint64_t fnv(uint64_t h, const void* p, size_t n) {
  const unsigned char* b = static_cast<const unsigned char*>(p);
  for (size_t i = 0; i < n; ++i) h = (h ^ b[i]) * 1099511628211ull;
  return h;
}

uint64_t structure_key(int dev, const std::vector<ResidentJob>& jobs) {
  uint64_t h = 1469598103934665603ull;
  h = fnv(h, &dev, sizeof(dev));
  for (const ResidentJob& j : jobs) {
    const uint64_t hdr[3] = {(uint64_t)j.n, (uint64_t)j.nparams, (uint64_t)j.nsets};
    h = fnv(h, hdr, sizeof(hdr));
    h = fnv(h, j.ops->data(), j.ops->size() * sizeof(AnsatzOp));
    h = fnv(h, j.groups, sizeof(HamTerms));
    h = fnv(h, j.zmask->data(), j.zmask->size() * sizeof(uint64_t));
    h = fnv(h, j.coef->data(), j.coef->size() * sizeof(double2));
  }
  return h;
}

std::mutex g_mu;
std::map<uint64_t, std::unique_ptr<Plan>>* g_plans = new std::map<uint64_t, std::unique_ptr<Plan>>();
constexpr size_t kMaxPlans = 16;

bool cuda_ok(cudaError_t e, const char* what, std::string& err) {
  if (e == cudaSuccess) return true;
  cudaGetLastError();
  err = std::string("resident executor: ") + what + ": " + cudaGetErrorString(e);
  return false;
}

template <class T>
bool upload(Plan& p, const std::vector<T>& v, T** out, std::string& err) {
  void* d = nullptr;
  if (!cuda_ok(device_alloc(&d, std::max<size_t>(v.size(), 1) * sizeof(T)), "cudaMalloc", err)) return false;
  p.dbufs.push_back(d);
  if (!v.empty() && !cuda_ok(cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice), "H2D", err))
    return false;
  *out = static_cast<T*>(d);
  return true;
}

// Bits of a stage for n index bits.  Three bits mean fewer stages; two bits
// keep twice the warps busy, which counts until the CTA's eight all have work.
// A whole gradient call (4 layers of Ry, Rz and a CX chain, TFIM), two bits /
// three: 8 qubits 107 / 133 us, 10: 138 / 158, 11: 214 / 201, 12: 380 / 355;
// with a barrier and a sweep per gate 172, 260, 374, 605 (of which 85 us are
// the call itself).  1024 sets at 12 qubits, where the FP64 units and shared
// memory bind: 4.1 -> 2.5 ms.
int stage_bits(int n) { return n >= kWideStageBits ? 3 : 2; }

// The gates of a circuit as stages of K bits.  A stage takes, in order, every
// gate whose target is one of its bits (the first K that come up) and that
// commutes past the gates left for later: diagonal uses of a qubit (a CX's
// control, CZ, Rz) commute with each other, all else on a common qubit does not.
void schedule(const ResidentJob& j, int K, std::vector<int4>& heads, std::vector<ResStep>& steps) {
  struct G {
    int kind, target, other, par;   // other: CX's control or CZ's second qubit, else -1
  };
  std::vector<G> left;
  for (const AnsatzOp& o : *j.ops) {
    switch (o.kind) {
      case GATE_RX: left.push_back({RES_RX, o.q0, -1, o.param}); break;
      case GATE_RY: left.push_back({RES_RY, o.q0, -1, o.param}); break;
      case GATE_RZ: case GATE_P: left.push_back({RES_RZ, o.q0, -1, o.param}); break;
      case GATE_U3:
        left.push_back({RES_RZ, o.q0, -1, o.param + 2});
        left.push_back({RES_RY, o.q0, -1, o.param});
        left.push_back({RES_RZ, o.q0, -1, o.param + 1});
        break;
      case GATE_H: left.push_back({RES_H, o.q0, -1, -1}); break;
      case GATE_X: left.push_back({RES_X, o.q0, -1, -1}); break;
      case GATE_SX: left.push_back({RES_SX, o.q0, -1, -1}); break;
      case GATE_CX: left.push_back({RES_CX, o.q1, o.q0, -1}); break;   // control q0
      default: left.push_back({RES_CZ, o.q0, o.q1, -1}); break;
    }
  }
  const int n = std::max(j.n, kMinBits);
  size_t first = 0;   // everything before is placed
  std::vector<G> in;
  while (first < left.size()) {
    // gates are taken from a window: what a gate far ahead could join is rare,
    // and the cost of planning stays linear
    const size_t end = std::min(left.size(), first + 512);
    uint32_t bits = 0, all = 0, diag = 0;   // the stage's bits; qubits with a waiting gate, with a waiting diagonal use
    int nrot = 0;
    in.clear();
    std::vector<G> wait;
    for (size_t i = first; i < end; ++i) {
      const G& g = left[i];
      const uint32_t t = 1u << g.target, o = g.other >= 0 ? 1u << g.other : 0u;
      const bool tdiag = g.kind == RES_RZ || g.kind == RES_CZ;
      const uint32_t dmask = o | (tdiag ? t : 0u), xmask = tdiag ? 0u : t;
      bool ok = !(dmask & all) && !(xmask & (all | diag)) && (int)in.size() < kStageSteps;
      if (ok && g.kind != RES_CZ && !(bits & t) && __builtin_popcount(bits) == K) ok = false;
      if (ok && g.kind <= RES_RZ) {
        if (nrot == kStageRots) ok = false;
        for (const G& x : in) ok = ok && !(x.kind <= RES_RZ && x.par == g.par);
      }
      if (!ok) {
        all |= xmask;
        diag |= dmask;
        wait.push_back(g);
        continue;
      }
      if (g.kind != RES_CZ) bits |= t;
      nrot += g.kind <= RES_RZ;
      in.push_back(g);
    }
    first = end - wait.size();   // what waits moves up behind what is placed
    std::copy(wait.begin(), wait.end(), left.begin() + first);
    for (int q = 0; q < n && __builtin_popcount(bits) < K; ++q) bits |= 1u << q;
    int local[32], pos = 0, packed = 0;
    for (int q = 0; q < 32; ++q) {
      local[q] = -1;
      if (bits >> q & 1) {
        packed |= q << (8 * pos);
        local[q] = pos++;
      }
    }
    const int pattern[3] = {0xAA, 0xCC, 0xF0};   // amplitudes whose local bit is set
    int r = 0;
    for (const G& g : in) {
      ResStep s = make_int4(g.kind * 4 + std::max(0, local[g.target]), 0, 0, 0);
      if (g.kind <= RES_RZ) {
        s.y = g.par;
        s.z = r++;
      } else if (g.kind >= RES_CX) {
        s.z = 0xFF;
        for (int q : {g.other, g.kind == RES_CZ ? g.target : g.other}) {
          if (local[q] >= 0) s.z &= pattern[local[q]];
          else s.y |= 1 << q;
        }
      }
      steps.push_back(s);
    }
    steps.resize((heads.size() + 1) * kStageSteps, make_int4(-1, 0, 0, 0));
    heads.push_back(make_int4((int)in.size(), nrot, packed, 0));
  }
}

std::unique_ptr<Plan> build(int dev, const std::vector<ResidentJob>& jobs, std::string& err) {
  std::unique_ptr<Plan> p(new Plan);
  p->dev = dev;
  std::vector<ResCirc> circs;
  std::vector<int2> items;
  std::vector<int4> heads;
  std::vector<ResStep> steps;
  std::vector<uint64_t> gx, tz;
  std::vector<int> gfirst;
  std::vector<double2> tc;
  std::vector<std::pair<double, int2>> order;
  int nmax = kMinBits, pmax = 1;
  for (size_t c = 0; c < jobs.size(); ++c) {
    const ResidentJob& j = jobs[c];
    ResCirc rc{};
    rc.n = std::max(j.n, kMinBits);
    rc.k = stage_bits(rc.n);
    rc.st0 = (int)heads.size();
    schedule(j, rc.k, heads, steps);
    rc.nst = (int)heads.size() - rc.st0;
    rc.nparams = j.nparams;
    rc.ngroups = j.groups->ngroups;
    rc.g0 = (int)gx.size();
    rc.t0 = (int)tz.size();
    rc.param0 = p->nparams_total;
    rc.e0 = p->nenergies;
    rc.grad0 = p->ngrads;
    for (int g = 0; g < rc.ngroups; ++g) {
      gx.push_back(j.groups->xmask[g]);
      gfirst.push_back(j.groups->first[g]);
    }
    gfirst.push_back(j.groups->first[rc.ngroups]);
    // gfirst is indexed by g0 + g with one closing entry per circuit: keep the
    // group arrays aligned by padding gx with the closing slot
    gx.push_back(0);
    tz.insert(tz.end(), j.zmask->begin(), j.zmask->end());
    tc.insert(tc.end(), j.coef->begin(), j.coef->end());
    p->nparams_total += j.nsets * (size_t)j.nparams;
    p->nenergies += j.nsets;
    p->ngrads += j.nsets * (size_t)j.nparams;
    nmax = std::max(nmax, rc.n);
    pmax = std::max(pmax, j.nparams);
    for (size_t s = 0; s < j.nsets; ++s)
      order.push_back({std::ldexp((double)(j.ops->size() + 1), j.n), make_int2((int)c, (int)s)});
    circs.push_back(rc);
  }
  // largest items first, ties in input order
  std::stable_sort(order.begin(), order.end(),
                   [](const std::pair<double, int2>& a, const std::pair<double, int2>& b) { return a.first > b.first; });
  for (auto& o : order) items.push_back(o.second);

  if (!cuda_ok(cudaSetDevice(dev), "cudaSetDevice", err) ||
      !cuda_ok(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking), "stream", err))
    return nullptr;
  ResCirc* d_circs;
  int2* d_items;
  int4* d_heads;
  ResStep* d_steps;
  uint64_t *d_gx, *d_tz;
  int* d_gfirst;
  double2* d_tc;
  if (!upload(*p, circs, &d_circs, err) || !upload(*p, items, &d_items, err) || !upload(*p, heads, &d_heads, err) ||
      !upload(*p, steps, &d_steps, err) ||
      !upload(*p, gx, &d_gx, err) || !upload(*p, gfirst, &d_gfirst, err) || !upload(*p, tz, &d_tz, err) ||
      !upload(*p, tc, &d_tc, err))
    return nullptr;
  std::vector<double> zeros_p(p->nparams_total), zeros_e(p->nenergies), zeros_g(p->ngrads);
  std::vector<int> zero_head(1, 0);
  double *d_params, *d_e, *d_g;
  int* d_head;
  if (!upload(*p, zeros_p, &d_params, err) || !upload(*p, zeros_e, &d_e, err) || !upload(*p, zeros_g, &d_g, err) ||
      !upload(*p, zero_head, &d_head, err))
    return nullptr;
  if (!cuda_ok(cudaMallocHost(&p->h_params, std::max<size_t>(p->nparams_total, 1) * 8), "pinned", err) ||
      !cuda_ok(cudaMallocHost(&p->h_e, std::max<size_t>(p->nenergies, 1) * 8), "pinned", err) ||
      !cuda_ok(cudaMallocHost(&p->h_g, std::max<size_t>(p->ngrads, 1) * 8), "pinned", err))
    return nullptr;

  const size_t smem = smem_bytes(nmax, pmax);
  if (!cuda_ok(cudaFuncSetAttribute(resident_adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "shared-memory limit", err))
    return nullptr;
  int per_sm = 0, sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!cuda_ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, resident_adjoint_kernel, kResThreads, smem),
               "occupancy", err))
    return nullptr;
  if (per_sm < 1) { err = "resident executor: a CTA does not fit an SM"; return nullptr; }
  const int grid = (int)std::min<size_t>(items.size(), (size_t)per_sm * sms);

  // capture: parameters up, queue head reset, the persistent launch, results down
  cudaGraph_t graph = nullptr;
  if (!cuda_ok(cudaStreamBeginCapture(p->stream, cudaStreamCaptureModeThreadLocal), "begin capture", err))
    return nullptr;
  cudaMemcpyAsync(d_params, p->h_params, std::max<size_t>(p->nparams_total, 1) * 8, cudaMemcpyHostToDevice, p->stream);
  cudaMemsetAsync(d_head, 0, sizeof(int), p->stream);
  resident_adjoint_kernel<<<grid, kResThreads, smem, p->stream>>>(d_circs, d_items, (int)items.size(), d_head, d_heads,
                                                                  d_steps, d_gx, d_gfirst, d_tz, d_tc, d_params, d_e,
                                                                  d_g, 1 << nmax, pmax);
  cudaMemcpyAsync(p->h_e, d_e, std::max<size_t>(p->nenergies, 1) * 8, cudaMemcpyDeviceToHost, p->stream);
  cudaMemcpyAsync(p->h_g, d_g, std::max<size_t>(p->ngrads, 1) * 8, cudaMemcpyDeviceToHost, p->stream);
  const cudaError_t ce = cudaStreamEndCapture(p->stream, &graph);
  if (!cuda_ok(ce, "end capture", err)) {
    if (graph) cudaGraphDestroy(graph);
    return nullptr;
  }
  const cudaError_t ie = cudaGraphInstantiate(&p->exec, graph, 0);
  cudaGraphDestroy(graph);
  if (!cuda_ok(ie, "graph instantiate", err)) return nullptr;
  return p;
}

}  // namespace

bool resident_run(int dev, const std::vector<ResidentJob>& jobs, std::string& err, double* host_ms) {
  if (jobs.empty()) return true;
  for (const ResidentJob& j : jobs)
    if (j.n < 1 || j.n > kResidentMaxQubits || j.nparams > kResidentMaxParams || !j.ops || !j.groups) {
      err = "resident executor: a circuit outside its limits";
      return false;
    }
  const auto t0 = std::chrono::steady_clock::now();
  std::lock_guard<std::mutex> g(g_mu);
  const uint64_t key = structure_key(dev, jobs);
  auto it = g_plans->find(key);
  if (it == g_plans->end()) {
    if (g_plans->size() >= kMaxPlans) g_plans->erase(g_plans->begin());
    std::unique_ptr<Plan> p = build(dev, jobs, err);
    if (!p) return false;
    it = g_plans->emplace(key, std::move(p)).first;
  }
  Plan& p = *it->second;
  size_t off = 0;
  for (const ResidentJob& j : jobs) {
    const size_t cnt = j.nsets * (size_t)j.nparams;
    if (cnt) std::memcpy(p.h_params + off, j.params, cnt * sizeof(double));
    off += cnt;
  }
  if (!cuda_ok(cudaSetDevice(dev), "cudaSetDevice", err) ||
      !cuda_ok(cudaGraphLaunch(p.exec, p.stream), "graph launch", err) ||
      !cuda_ok(cudaStreamSynchronize(p.stream), "sync", err))
    return false;
  size_t eo = 0, go = 0;
  for (const ResidentJob& j : jobs) {
    for (size_t s = 0; s < j.nsets; ++s) {
      if (j.energy_out) j.energy_out[s] = p.h_e[eo + s];
      if (j.grad_out)
        std::memcpy(j.grad_out + s * (size_t)j.nparams, p.h_g + go + s * (size_t)j.nparams, j.nparams * sizeof(double));
    }
    eo += j.nsets;
    go += j.nsets * (size_t)j.nparams;
  }
  if (host_ms) *host_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return true;
}

void resident_release() {
  std::lock_guard<std::mutex> g(g_mu);
  g_plans->clear();
}

}  // namespace iqb
