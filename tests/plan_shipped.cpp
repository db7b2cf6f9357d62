// plan_shipped.cpp -- TEST ONLY.  The plans the library runs -- steady
// decomposition of state programs, framed single-set gradients, the diagonals of
// each register stage merged -- executed on the CPU by plan_emulator.cpp's tile
// emulation, which knows every operation but the merged ones.
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
