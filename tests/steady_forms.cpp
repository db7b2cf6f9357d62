// CPU checks of the angle-independent forms: decompose_one_qubit_ops in its
// steady mode and the Pauli frame of an ansatz, by dense application of the
// operation lists.  Built and called by tests/test_steady_forms.py.
#include <cmath>
#include <complex>
#include <random>
#include <string>
#include <vector>

#include "../invariantq_b200/csrc/iq_plan.h"

using namespace iqb;
using cd = std::complex<double>;

namespace iqb {
std::string jit_pass_key(const PassDesc& d, int min_blocks, int threads, bool set_mode, bool narrow);
}

namespace {

void apply(std::vector<cd>& v, const SchedOp& o, const std::vector<cplx64>& pool) {
  const int d = 1 << o.k;
  const cplx64* m = pool.data() + o.dense;
  std::vector<cd> in(d);
  for (size_t x = 0; x < v.size(); ++x) {
    bool first = true;
    for (int j = 0; j < o.k; ++j) first = first && !((x >> o.q[j]) & 1);
    if (!first) continue;
    auto at = [&](int l) {
      size_t y = x;
      for (int j = 0; j < o.k; ++j)
        if ((l >> j) & 1) y |= (size_t)1 << o.q[j];
      return y;
    };
    for (int l = 0; l < d; ++l) in[l] = v[at(l)];
    for (int r = 0; r < d; ++r) {
      cd s = 0.0;
      for (int c = 0; c < d; ++c) s += cd(m[r * d + c].re, m[r * d + c].im) * in[c];
      v[at(r)] = s;
    }
  }
}

void push(std::vector<SchedOp>& ops, std::vector<cplx64>& pool, int k, const int* q, const cd* m) {
  SchedOp o{};
  o.k = (uint8_t)k;
  for (int j = 0; j < k; ++j) o.q[j] = (uint8_t)q[j];
  const int d = 1 << k;
  o.dense = o.mat = (uint32_t)pool.size();
  for (int i = 0; i < d * d; ++i) pool.push_back({m[i].real(), m[i].imag()});
  double ph[8];
  uint8_t perm = 0, unit = 0;
  if (k <= 2 && classify_monomial(reinterpret_cast<const double*>(m), k, &perm, ph, &unit)) {
    o.mono = 1;
    o.perm = perm;
    o.unit = unit;
    o.mat = (uint32_t)pool.size();
    for (int i = 0; i < d; ++i) pool.push_back({ph[2 * i], ph[2 * i + 1]});
  } else if (k == 2) {
    o.xpat = (uint8_t)classify_xpattern(reinterpret_cast<const double*>(m));
  }
  ops.push_back(o);
}

}  // namespace

extern "C" {

// A random circuit of `count` operations on n bits: the largest difference
// between its list and the list's steady form on a random vector.
double steady_error(int n, int count, int seed) {
  std::mt19937_64 r(seed);
  std::uniform_real_distribution<double> u(0.0, 2.0 * M_PI);
  std::normal_distribution<double> g;
  std::vector<SchedOp> ops;
  std::vector<cplx64> pool;
  for (int i = 0; i < count; ++i) {
    int q[3] = {(int)(r() % n), 0, 0};
    do q[1] = (int)(r() % n); while (q[1] == q[0]);
    do q[2] = (int)(r() % n); while (q[2] == q[0] || q[2] == q[1]);
    const double t = u(r), a = u(r), b = u(r), c = std::cos(t / 2), s = std::sin(t / 2);
    const cd ea = std::polar(1.0, a), eb = std::polar(1.0, b);
    cd m[64] = {};
    switch (r() % 11) {
      case 0: case 1: case 2: m[0] = c; m[1] = -eb * s; m[2] = ea * s; m[3] = ea * eb * c; push(ops, pool, 1, q, m); break;
      case 3: m[1] = ea; m[2] = eb; push(ops, pool, 1, q, m); break;                    // X with phases
      case 4: m[0] = ea; m[3] = eb; push(ops, pool, 1, q, m); break;
      case 5: m[0] = m[5] = m[11] = m[14] = 1.0; push(ops, pool, 2, q, m); break;       // CX
      case 6: m[0] = m[5] = m[10] = 1.0; m[15] = -1.0; push(ops, pool, 2, q, m); break; // CZ
      case 7: m[0] = ea; m[6] = eb; m[9] = 1.0; m[15] = ea; push(ops, pool, 2, q, m); break;
      case 8:   // a random permutation with phases
        { int p[4] = {0, 1, 2, 3};
          for (int k = 3; k > 0; --k) std::swap(p[k], p[r() % (k + 1)]);
          for (int k = 0; k < 4; ++k) m[4 * k + p[k]] = std::polar(1.0, u(r));
          push(ops, pool, 2, q, m); }
        break;
      case 9:   // a channel-shaped operation, or a damping diagonal
        if (r() & 1) { m[0] = 0.9; m[3] = 0.2; m[12] = 0.1; m[15] = 0.8; m[5] = 0.7; m[10] = 0.6; }
        else { m[0] = 1.0; m[5] = 0.9; m[10] = 0.8; m[15] = 0.7; }
        push(ops, pool, 2, q, m);
        break;
      default: {
        const int k = 2 + (int)(r() & 1), d = 1 << k;
        for (int j = 0; j < d * d; ++j) m[j] = cd(g(r), g(r)) / std::sqrt(2.0 * d);
        push(ops, pool, k, q, m);
      }
    }
  }
  std::vector<cd> v((size_t)1 << n), w;
  for (auto& x : v) x = cd(g(r), g(r));
  w = v;
  for (const SchedOp& o : ops) apply(v, o, pool);
  decompose_one_qubit_ops(ops, pool, DECOMP_STEADY);
  for (const SchedOp& o : ops) apply(w, o, pool);
  double e = 0.0, s = 0.0;
  for (size_t i = 0; i < v.size(); ++i) {
    e = std::max(e, std::abs(v[i] - w[i]));
    s = std::max(s, std::abs(v[i]));
  }
  return e / s;
}

// The frame of a random ansatz: the largest difference between |<basis|psi>| of
// the circuit and of X^x Z^z times the frame's circuit, phase aligned.
double frame_error(int n, int count, int seed) {
  std::mt19937_64 r(seed);
  std::uniform_real_distribution<double> u(0.0, 2.0 * M_PI);
  std::vector<AnsatzOp> ops;
  std::vector<double> th;
  for (int i = 0; i < count; ++i) {
    const int kind = 1 + (int)(r() % 10), a = (int)(r() % n);
    int b;
    do b = (int)(r() % n); while (b == a);
    const bool two = kind == GATE_CZ || kind == GATE_CX;
    int par = -1;
    if (kind <= GATE_P) {
      par = (int)th.size();
      for (int k = 0; k < (kind == GATE_U3 ? 3 : 1); ++k) th.push_back(u(r));
    }
    ops.push_back({kind, a, two ? b : -1, par});
  }
  std::vector<SchedOp> plain, framed;
  std::vector<cplx64> p0, p1;
  PauliFrame f;
  pauli_frame(ops, th.data(), f);
  ansatz_forward(n, ops, th.data(), plain, p0);
  ansatz_forward(n, ops, th.data(), framed, p1, true, &f);
  std::vector<cd> v((size_t)1 << n), w((size_t)1 << n), z((size_t)1 << n);
  v[0] = w[0] = 1.0;
  for (const SchedOp& o : plain) apply(v, o, p0);
  for (const SchedOp& o : framed) apply(w, o, p1);
  for (size_t x = 0; x < w.size(); ++x) z[x ^ f.x] = (__builtin_popcountll(x & f.z) & 1) ? -w[x] : w[x];
  cd overlap = 0.0;
  for (size_t x = 0; x < v.size(); ++x) overlap += std::conj(z[x]) * v[x];
  return std::abs(std::abs(overlap) - 1.0);
}

// Fingerprint of the planned passes' structure (what kernels are compiled for):
// kind 0 a U3 + CX brick-wall, 1 / 2 the forward / backward of an RY RZ CZ-ring
// ansatz, with angles from `seed`.
uint64_t structure(int kind, int n, int depth, int seed) {
  std::mt19937_64 r(seed);
  std::uniform_real_distribution<double> u(0.0, 2.0 * M_PI);
  std::vector<SchedOp> ops;
  std::vector<cplx64> pool;
  SchedParams p{};
  p.nbits = n;
  p.M = 12;
  p.c = 4;
  p.R = 4;
  p.max_stages = 8;
  p.budget = 160;
  if (kind == 0) {
    for (int l = 0; l < depth; ++l) {
      for (int q = 0; q < n; ++q) {
        const double t = u(r), c = std::cos(t / 2), s = std::sin(t / 2);
        const cd ea = std::polar(1.0, u(r)), eb = std::polar(1.0, u(r));
        const cd m[4] = {c, -eb * s, ea * s, ea * eb * c};
        push(ops, pool, 1, &q, m);
      }
      for (int q = l % 2; q + 1 < n; q += 2) {
        cd m[16] = {};
        m[0] = m[5] = m[11] = m[14] = 1.0;
        const int qq[2] = {q + 1, q};
        push(ops, pool, 2, qq, m);
      }
    }
    ops = fuse_two_qubit_blocks(ops, pool, true);
    decompose_one_qubit_ops(ops, pool, DECOMP_STEADY);
    normalize_one_qubit_ops(ops, pool);
  } else {
    std::vector<AnsatzOp> a;
    std::vector<double> th;
    for (int l = 0; l < depth; ++l) {
      for (int g : {GATE_RY, GATE_RZ})
        for (int q = 0; q < n; ++q) {
          a.push_back({g, q, -1, (int)th.size()});
          th.push_back(u(r));
        }
      for (int q = 0; q < n; ++q) a.push_back({GATE_CZ, q, (q + 1) % n, -1});
    }
    AdjointOps j;
    adjoint_ops(n, a, th.data(), true, true, true, j, true);
    ops = kind == 1 ? j.fw : j.bw;
    p.nbits += kind - 1;
  }
  std::vector<PassPlan> plans;
  std::string err;
  if (plan_passes(p, ops, plans, err) < 0) return 0;
  merge_stage_diagonals(plans, ops);
  PackRecipe rec;
  pack_recipe(plans, rec);
  uint64_t h = 1469598103934665603ull;
  auto put = [&](const std::string& k) {
    for (unsigned char ch : k) h = (h ^ ch) * 1099511628211ull;
  };
  for (const PassPlan& pl : plans) put(jit_pass_key(pl.desc, 3, 128, kind != 0, false));
  return h;
}

}  // extern "C"
