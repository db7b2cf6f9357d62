// plan_shipped.cpp -- TEST ONLY.  The plans the library runs -- steady
// decomposition of state programs, framed single-set gradients, the diagonals of
// each register stage merged -- executed on the CPU by plan_emulator.cpp's tile
// emulation, which knows every operation but the merged ones.
#include <cmath>
#include <random>

#include "plan_emulator.cpp"

namespace {

// one merged operation (OP_DGR, OP_GDZ) of stage s on a resident tile
void run_merged_op(Emu& e, const PassDesc& P, const StageDesc& sd, const OpDesc& od, std::vector<cd>& tile) {
  const int R = P.R, NV = 1 << R;
  for (uint32_t u = 0; u < (1u << sd.nt); ++u)
    for (uint32_t L = 0; L < 8; ++L) {
      uint32_t base = 0;
      for (int i = 0; i < sd.nt; ++i) base |= ((u >> i) & 1u) << sd.tb[i];
      for (int i = 0; i < 3; ++i) base |= ((L >> i) & 1u) << sd.lane[i];
      auto at = [&](int v) -> cd& {
        uint32_t o = base;
        for (int i = 0; i < R; ++i)
          if ((v >> i) & 1) o |= 1u << sd.S[i];
        return tile[swz(o)];
      };
      if (od.kind == OP_DGR) {
        for (int v = 0; v < NV; ++v) {
          const cd m = e.mat(od.mat, v & od.flags);
          const bool unit = (od.gidx >> v) & 1, neg = (od.gidx >> (16 + v)) & 1;
          // what the specialised kernels leave out has to be exactly that, and a row's entry that of its masked index
          if ((unit && m != 1.0) || (neg && m != -1.0) || e.mat(od.mat, v) != m) e.err = "merged diagonal: entry and flags disagree";
          if (!unit) at(v) *= m;
        }
        continue;
      }
      int term = (int)od.gidx;
      for (int b = 1; b < R; ++b) {
        if (!((od.flags >> b) & 1)) continue;
        const uint32_t t = P.grad_term[term++];
        for (int v = 0; v < NV; v += 2) {
          const double z = (std::conj(at(v | 1)) * at(v)).imag();
          e.grads[t] += ((v >> b) & 1) ? -z : z;
        }
      }
    }
}

struct MergedCounts { int dgr = 0, gdz = 0, passes = 0, stages = 0; };

// plan, merge and pack `ops` as the library does and run every pass on e.state
bool run_merged(Emu& e, const std::vector<SchedOp>& ops, SchedParams p, int gap, std::vector<PassPlan>& plans,
                MergedCounts& mc) {
  p.nbits = gap ? gap : e.nbits;
  if (plan_passes(p, ops, plans, e.err) < 0) return false;
  merge_stage_diagonals(plans, ops);
  for (PassPlan& pl : plans) pl.desc.gap = (uint8_t)gap;
  std::vector<cplx64> packed;
  pack_pass_matrices(plans, reinterpret_cast<const cplx64*>(e.pool.data()), packed);
  e.pool.assign(reinterpret_cast<const cd*>(packed.data()), reinterpret_cast<const cd*>(packed.data()) + packed.size());
  for (const PassPlan& pl : plans) {
    const PassDesc& P = pl.desc;
    e.blk = P.mat_base;
    ++mc.passes;
    mc.stages += P.nstages;
    for (uint32_t o = 0; o < P.nops; ++o) {
      mc.dgr += P.ops[o].kind == OP_DGR;
      mc.gdz += P.ops[o].kind == OP_GDZ;
    }
    std::vector<cd> tile((size_t)1 << P.M);
    std::vector<uint8_t> seen((size_t)1 << e.nbits, 0);
    PassDesc one = P;
    for (uint64_t t = 0; t < P.ntiles && e.err.empty(); ++t) {
      if (!e.copy_tile(P, t, tile, true, seen)) return false;
      for (int s = 0; s < P.nstages && e.err.empty(); ++s)
        for (int o = P.st[s].op0; o < P.st[s].op1 && e.err.empty(); ++o) {
          if (P.ops[o].kind == OP_DGR || P.ops[o].kind == OP_GDZ) {
            run_merged_op(e, P, P.st[s], P.ops[o], tile);
            continue;
          }
          one.st[s].op0 = (uint16_t)o;
          one.st[s].op1 = (uint16_t)(o + 1);
          e.run_stage(one, s, tile);
        }
      if (!e.err.empty() || !e.copy_tile(P, t, tile, false, seen)) return false;
    }
    for (size_t i = 0; i < seen.size(); ++i)
      if (seen[i] != ((!gap || !((i >> gap) & 1)) ? 1 : 0)) {
        e.err = "a pass does not cover its part of the array exactly";
        return false;
      }
  }
  return e.err.empty();
}

SchedParams sched_params(int M, int c, int R, int max_stages, double budget) {
  SchedParams p{};
  p.M = M;
  p.c = c;
  p.R = R;
  p.max_stages = max_stages;
  p.budget = budget;
  return p;
}

void set_pool(Emu& e, const std::vector<cplx64>& pool) {
  e.pool.assign(reinterpret_cast<const cd*>(pool.data()), reinterpret_cast<const cd*>(pool.data()) + pool.size());
}

}  // namespace

// Operations (LSB-first qubit lists, dense matrices) on `state`, planned as state
// programs for the specialised kernels are.  counts: passes, stages, OP_DGR.
extern "C" int shipped_apply(int nbits, int M, int c, int R, int max_stages, double budget, int nops, const int* ks,
                             const int* qs, const double* mats, const long long* mat_off, double* state, int* counts,
                             char* errbuf, int errlen) {
  std::vector<cplx64> pool;
  std::vector<SchedOp> ops;
  for (int i = 0; i < nops; ++i) {
    SchedOp o{};
    o.k = (uint8_t)ks[i];
    for (int j = 0; j < ks[i]; ++j) o.q[j] = (uint8_t)qs[i * 5 + j];
    const int d = 1 << ks[i];
    const double* m = mats + 2 * mat_off[i];
    o.mat = o.dense = (uint32_t)pool.size();
    for (int j = 0; j < d * d; ++j) pool.push_back({m[2 * j], m[2 * j + 1]});
    double ph[8];
    if (ks[i] <= 2 && classify_monomial(m, ks[i], &o.perm, ph, &o.unit)) {
      o.mono = 1;
      o.mat = (uint32_t)pool.size();
      for (int j = 0; j < d; ++j) pool.push_back({ph[2 * j], ph[2 * j + 1]});
    } else if (ks[i] == 2) {
      o.xpat = (uint8_t)classify_xpattern(m);
    }
    ops.push_back(o);
  }
  ops = fuse_two_qubit_blocks(ops, pool, true);
  decompose_one_qubit_ops(ops, pool, DECOMP_STEADY);
  normalize_one_qubit_ops(ops, pool);
  Emu e;
  e.nbits = nbits;
  e.state = reinterpret_cast<cd*>(state);
  set_pool(e, pool);
  std::vector<PassPlan> plans;
  MergedCounts mc;
  if (!run_merged(e, ops, sched_params(M, c, R, max_stages, budget), 0, plans, mc)) {
    snprintf(errbuf, errlen, "%s", e.err.c_str());
    return -1;
  }
  counts[0] = mc.passes;
  counts[1] = mc.stages;
  counts[2] = mc.dgr;
  return 0;
}

// Rounding on the host alone: a U3 + CX brick-wall's gates and the steady list
// made of them, both applied to a basis state in long double.  out: the norm of
// the difference, the difference of the squared norms.
extern "C" void host_rounding(int n, int depth, int seed, double* out) {
  using cl = std::complex<long double>;
  std::mt19937_64 r(seed);
  std::uniform_real_distribution<double> u(0.0, 2.0 * M_PI);
  std::vector<SchedOp> ops;
  std::vector<cplx64> pool;
  auto push = [&](std::initializer_list<int> q, const cd* m) {
    SchedOp o{};
    for (int b : q) o.q[o.k++] = (uint8_t)b;
    const int d = 1 << o.k;
    o.dense = o.mat = (uint32_t)pool.size();
    for (int i = 0; i < d * d; ++i) pool.push_back({m[i].real(), m[i].imag()});
    double ph[8];
    if (classify_monomial(reinterpret_cast<const double*>(m), o.k, &o.perm, ph, &o.unit)) {
      o.mono = 1;
      o.mat = (uint32_t)pool.size();
      for (int i = 0; i < d; ++i) pool.push_back({ph[2 * i], ph[2 * i + 1]});
    }
    ops.push_back(o);
  };
  for (int l = 0; l < depth; ++l) {
    for (int q = 0; q < n; ++q) {
      const double t = u(r), c = std::cos(t / 2), s = std::sin(t / 2);
      const cd ea = std::polar(1.0, u(r)), eb = std::polar(1.0, u(r));
      const cd m[4] = {c, -eb * s, ea * s, ea * eb * c};
      push({q}, m);
    }
    cd cx[16] = {};
    cx[0] = cx[5] = cx[11] = cx[14] = 1.0;
    for (int q = l % 2; q + 1 < n; q += 2) push({q + 1, q}, cx);
  }
  auto run = [&](std::vector<cl>& v) {
    for (const SchedOp& o : ops) {
      const int d = 1 << o.k;
      for (size_t x = 0; x < v.size(); ++x) {
        size_t idx[4];
        bool lead = true;
        for (int l = 0; l < d; ++l) {
          idx[l] = x;
          for (int j = 0; j < o.k; ++j) {
            lead = lead && !((x >> o.q[j]) & 1);
            if ((l >> j) & 1) idx[l] |= (size_t)1 << o.q[j];
          }
        }
        if (!lead) continue;
        cl in[4];
        for (int l = 0; l < d; ++l) in[l] = v[idx[l]];
        for (int row = 0; row < d; ++row) {
          cl s = 0.0L;
          for (int c = 0; c < d; ++c) s += cl(pool[o.dense + row * d + c].re, pool[o.dense + row * d + c].im) * in[c];
          v[idx[row]] = s;
        }
      }
    }
  };
  std::vector<cl> v((size_t)1 << n), w((size_t)1 << n);
  v[0] = w[0] = 1.0L;
  run(v);
  ops = fuse_two_qubit_blocks(ops, pool, true);
  decompose_one_qubit_ops(ops, pool, DECOMP_STEADY);
  normalize_one_qubit_ops(ops, pool);
  run(w);
  long double e = 0.0L, dn = 0.0L;
  for (size_t x = 0; x < v.size(); ++x) {
    e += std::norm(v[x] - w[x]);
    dn += std::norm(w[x]) - std::norm(v[x]);
  }
  out[0] = (double)std::sqrt(e);
  out[1] = (double)dn;
}

// The largest error, in units of 2^-53, of a component of merged entries that are
// products of `count` phases (of modulus 1) from `seed`
extern "C" double merged_entry_error(int count, int seed) {
  std::mt19937_64 r(seed);
  std::uniform_real_distribution<double> u(0.0, 2.0 * M_PI);
  std::vector<cplx64> pool(64), out(256);
  for (cplx64& p : pool) {
    const double t = u(r);
    p = {std::cos(t), std::sin(t)};
  }
  PackRecipe rec;
  std::vector<std::vector<uint32_t>> factors(out.size());
  for (uint32_t i = 0; i < out.size(); ++i) {
    factors[i].push_back((uint32_t)(r() % pool.size()));
    rec.base.push_back(factors[i][0]);
    for (int k = 1; k < count; ++k) {
      factors[i].push_back((uint32_t)(r() % pool.size()));
      rec.mults.push_back({i, factors[i].back()});
    }
  }
  rec.fill(pool.data(), out.data());
  double worst = 0.0;
  for (size_t i = 0; i < out.size(); ++i) {
    __float128 re = 1, im = 0;
    for (uint32_t f : factors[i]) {
      const __float128 t = re * pool[f].re - im * pool[f].im;
      im = re * pool[f].im + im * pool[f].re;
      re = t;
    }
    worst = std::max({worst, (double)std::fabs((double)(re - out[i].re)), (double)std::fabs((double)(im - out[i].im))});
  }
  return worst * 0x1p53;
}

// Energy and gradient of an ansatz with one parameter set (n >= 7), through the
// operation lists, frame, plans and merged stages the executor runs.
// counts: OP_DGR and OP_GDZ operations, scalar operations of the backward list.
extern "C" int shipped_adjoint(int n, int nops, const int* kinds, const int* q0, const int* q1, const int* pidx,
                               const double* params, int nterms, const double* coeffs, const char* paulis, int M, int c,
                               int R, int max_stages, double budget, double* energy, double* grad, int nparams,
                               int* counts, char* errbuf, int errlen) {
  std::vector<AnsatzOp> ops(nops);
  for (int i = 0; i < nops; ++i) ops[i] = {kinds[i], q0[i], q1[i], pidx[i]};
  std::string err;
  if (ansatz_check(n, ops, err) < 0) {
    snprintf(errbuf, errlen, "%s", err.c_str());
    return -1;
  }
  const SchedParams p = sched_params(M, c, R, max_stages, budget);
  AdjointOps jo;
  adjoint_ops(n, ops, params, true, true, true, jo, true);
  const uint64_t dim = 1ULL << n;
  std::vector<cd> joint(2 * dim, 0.0);
  joint[0] = 1.0;
  MergedCounts mc;
  std::vector<PassPlan> fwp, bwp;
  Emu f, b;
  f.nbits = b.nbits = n + 1;
  f.state = b.state = joint.data();
  set_pool(f, jo.fpool);
  set_pool(b, jo.bpool);
  b.grads.assign(jo.grad_param.size(), 0.0);
  bool ok = run_merged(f, jo.fw, p, n, fwp, mc);
  // lambda = F H F psi, F = X^x Z^z the set's frame: strings that do not commute with it change sign
  cd en = 0.0;
  for (int t = 0; ok && t < nterms; ++t) {
    uint64_t xm = 0, zm = 0;
    cd ip = 1.0;
    for (int q = 0; q < n; ++q) {
      const char ch = paulis[t * n + q];
      if (ch == 'X' || ch == 'Y') xm |= 1ULL << q;
      if (ch == 'Z' || ch == 'Y') zm |= 1ULL << q;
      if (ch == 'Y') ip *= cd(0, 1);
    }
    const bool flip = (__builtin_popcountll(zm & jo.frame.x) + __builtin_popcountll(xm & jo.frame.z)) & 1;
    for (uint64_t j = 0; j < dim; ++j) {
      const uint64_t i = j ^ xm;
      const double sg = ((__builtin_popcountll(i & zm) & 1) != (flip ? 1 : 0)) ? -1.0 : 1.0;
      joint[dim + j] += coeffs[t] * ip * sg * joint[i];
    }
  }
  for (uint64_t x = 0; x < dim; ++x) en += std::conj(joint[x]) * joint[dim + x];
  *energy = en.real();
  ok = ok && run_merged(b, jo.bw, p, 0, bwp, mc);
  std::vector<double> scale;
  exec_grad_scales(&bwp, jo.bw, scale);
  if (ok && (scale.size() != jo.grad_param.size() || jo.grad_sign.size() != scale.size())) {
    ok = false;
    b.err = "gradient scales and signs do not match the terms";
  }
  if (!ok) {
    snprintf(errbuf, errlen, "%s%s", f.err.c_str(), b.err.c_str());
    return -1;
  }
  for (int i = 0; i < nparams; ++i) grad[i] = 0.0;
  for (size_t t = 0; t < scale.size(); ++t) grad[jo.grad_param[t]] += b.grads[t] * scale[t] * jo.grad_sign[t];
  counts[0] = mc.dgr;
  counts[1] = mc.gdz;
  counts[2] = 0;
  for (const SchedOp& o : jo.bw) counts[2] += o.smul != 0.0 && !o.grad;
  return 0;
}

// Fingerprint of the plans (what shapes and kernels are found by) of one
// parameter set's forward or backward list; 0 on an error.
extern "C" unsigned long long shipped_structure(int n, int nops, const int* kinds, const int* q0, const int* q1,
                                                const int* pidx, const double* params, int backward) {
  std::vector<AnsatzOp> ops(nops);
  for (int i = 0; i < nops; ++i) ops[i] = {kinds[i], q0[i], q1[i], pidx[i]};
  std::string err;
  if (ansatz_check(n, ops, err) < 0) return 0;
  AdjointOps jo;
  adjoint_ops(n, ops, params, true, true, true, jo, true);
  const std::vector<SchedOp>& list = backward ? jo.bw : jo.fw;
  SchedParams p = sched_params(12, 4, 4, 8, 160.0);
  p.nbits = n + (backward ? 1 : 0);
  std::vector<PassPlan> plans;
  if (plan_passes(p, list, plans, err) < 0) return 0;
  merge_stage_diagonals(plans, list);
  PackRecipe rec;
  pack_recipe(plans, rec);
  uint64_t h = 1469598103934665603ull;
  for (const PassPlan& pl : plans)
    for (unsigned char ch : jit_pass_key(pl.desc, 3, 128, true, false)) h = (h ^ ch) * 1099511628211ull;
  return h;
}

// For every pass of a state program's plan: log2 of its tile's copies, and
// whether it runs in the pair pipeline.  Returns the passes, -1 on an error.
extern "C" int shipped_forms(int nbits, int nops, const int* ks, const int* qs, const double* mats,
                             const long long* mat_off, int* boxes, int* pair, int max_passes) {
  std::vector<cplx64> pool;
  std::vector<SchedOp> ops;
  for (int i = 0; i < nops; ++i) {
    SchedOp o{};
    o.k = (uint8_t)ks[i];
    for (int j = 0; j < ks[i]; ++j) o.q[j] = (uint8_t)qs[i * 5 + j];
    const int d = 1 << ks[i];
    const double* m = mats + 2 * mat_off[i];
    o.mat = o.dense = (uint32_t)pool.size();
    for (int j = 0; j < d * d; ++j) pool.push_back({m[2 * j], m[2 * j + 1]});
    double ph[8];
    if (ks[i] <= 2 && classify_monomial(m, ks[i], &o.perm, ph, &o.unit)) {
      o.mono = 1;
      o.mat = (uint32_t)pool.size();
      for (int j = 0; j < d; ++j) pool.push_back({ph[2 * j], ph[2 * j + 1]});
    }
    ops.push_back(o);
  }
  ops = fuse_two_qubit_blocks(ops, pool, true);
  decompose_one_qubit_ops(ops, pool, DECOMP_STEADY);
  normalize_one_qubit_ops(ops, pool);
  SchedParams p = sched_params(12, 4, 4, 8, 160.0);
  p.nbits = nbits;
  std::vector<PassPlan> plans;
  std::string err;
  if (plan_passes(p, ops, plans, err) < 0 || (int)plans.size() > max_passes) return -1;
  merge_stage_diagonals(plans, ops);
  for (size_t i = 0; i < plans.size(); ++i) {
    const PassDesc& d = plans[i].desc;
    boxes[i] = d.nH - d.nbox;
    pair[i] = pair_form_fits(d) && jit_pass_threads(d, kPairForm) == kPairForm;
  }
  return (int)plans.size();
}
