// iq_sched.cpp -- host-side gate scheduler: turns the queue of gates and
// channels recorded through the C ABI into tile passes (see iq_plan.h).
//
// The reference applies every gate as its own sweep over the state
// (core/src/statevector.cpp:26-152, one OpenMP loop per call).  Here the
// queued operations are grouped greedily, in dependency order, into passes
// whose operations all act on the M index bits a tile holds, so a group of
// gates costs one read and one write of the array.  Inside a pass the
// operations are split into register stages (R register slots + 3 lane bits).
// Operations are applied in queue order per qubit, so the result is the same
// product of matrices the reference applies one call at a time.
#include "iq_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <array>
#include <complex>
#include <set>

namespace iqb {

// complex elements of an operation's matrix data (dense 4^k, monomial 2^k phases)
int op_mat_elems(const SchedOp& op) {
  if (op.grad) return 4;
  return op.mono ? (1 << op.k) : (1 << (2 * op.k));
}

double op_cost(const SchedOp& op, double grad_cost) {
  if (op.grad) return grad_cost;   // 2x2 on both halves plus the gradient products
  if (op.mono) {
    if (op.unit) return 0.25;
    const int rows = 1 << op.k;
    const int nonunit = rows - __builtin_popcount(op.urows & ((1u << rows) - 1));
    return 4.0 * nonunit / rows;
  }
  if (op.rot) return 2.0;
  if (op.norm) return 6.0;
  if (op.realm && op.k == 1) return 4.0;
  if (op.xpat) return ((op.xpat & XPAT_CORNERS_REAL) ? 2.0 : 4.0) + ((op.xpat & XPAT_MIDDLE_REAL) ? 1.0 : 2.0);
  return 4.0 * double(1u << op.k);
}

int classify_monomial(const double* m, int k, uint8_t* perm, double* phases, uint8_t* unit) {
  if (k < 1 || k > 2) return 0;
  const int d = 1 << k;
  int colcount[4] = {0, 0, 0, 0};
  uint8_t p = 0;
  uint8_t u = 1;
  for (int r = 0; r < d; ++r) {
    int nz = -1;
    for (int c = 0; c < d; ++c) {
      const double re = m[2 * (r * d + c)], im = m[2 * (r * d + c) + 1];
      if (re != 0.0 || im != 0.0) {
        if (nz >= 0) return 0;
        nz = c;
      }
    }
    if (nz < 0) return 0;
    colcount[nz]++;
    p |= uint8_t(nz << (2 * r));
    phases[2 * r] = m[2 * (r * d + nz)];
    phases[2 * r + 1] = m[2 * (r * d + nz) + 1];
    if (phases[2 * r] != 1.0 || phases[2 * r + 1] != 0.0) u = 0;
  }
  for (int c = 0; c < d; ++c)
    if (colcount[c] != 1) return 0;
  *perm = p;
  *unit = u;
  return 1;
}

int classify_xpattern(const double* m) {
  bool corners_real = true, middle_real = true;
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      const double re = m[2 * (r * 4 + c)], im = m[2 * (r * 4 + c) + 1];
      const bool corner = (r == 0 || r == 3) && (c == 0 || c == 3);
      const bool middle = r == c && (r == 1 || r == 2);
      if (!corner && !middle && (re != 0.0 || im != 0.0)) return 0;
      if (corner && im != 0.0) corners_real = false;
      if (middle && im != 0.0) middle_real = false;
    }
  return 1 | (corners_real ? XPAT_CORNERS_REAL : 0) | (middle_real ? XPAT_MIDDLE_REAL : 0);
}

namespace {

struct StageBits {                 // what placing an operation reads and changes (copied for each trial)
  int S[kMaxK];
  int nS = 0;
  uint64_t lanereq = 0;            // bits that 1q lane operations of this stage act on
  bool dk = false;                 // holds one dense k>=3 block; closed
};
struct Stage : StageBits {
  std::vector<int> ops;
};

struct PassBuilder {
  const SchedParams& p;
  int c;
  std::vector<Stage> stages;
  bool allow_new = true;   // false: an operation joins the current stage or waits
  explicit PassBuilder(const SchedParams& pp, int cc) : p(pp), c(cc) {}

  static bool inS(const StageBits& s, int b) {
    for (int i = 0; i < s.nS; ++i)
      if (s.S[i] == b) return true;
    return false;
  }
  int lowcount(const StageBits& s) const {
    int n = 0;
    for (int i = 0; i < s.nS; ++i) n += s.S[i] < c;
    return n;
  }
  // Chunk bits a stage may hold in slots: c - 3 keeps three chunk bits free for
  // lane operations.  A stage without lane operations may take one more: its
  // lanes can then use the first tile bit above the chunk, whose swizzled
  // image also has a low bit set, so the octet's accesses can stay on eight
  // bank groups (the lane choice below takes the best rank it finds).
  int lowlimit(const StageBits& s, bool no_lanes_after) const {
    return c - kLaneBits + ((no_lanes_after && s.lanereq == 0) ? 1 : 0);
  }
  // Whether a stage without lane operations whose slots also take the nn bits
  // `add` keeps three lane candidates with independent swizzle images: the
  // low three bits of swz(1 << j) are bit j mod 3 for tile-local j < 6 and 0
  // above, so each class {k, k + 3} (k = 0, 1, 2) needs a member outside the
  // slots.  Tile-local bits >= c are high tile bits chosen when the pass is
  // finalised; physical bit j stands in for them (it is the one they are when
  // it is local in the pass).
  bool lanes_feasible(const StageBits& s, const int* add, int nn) const {
    for (int k = 0; k < 3; ++k) {
      bool free_member = false;
      for (int j = k; j < 6 && !free_member; j += 3) {
        // j >= c: the high tile bit H[j - c] is at least physical bit j, and is
        // that bit whenever it is local; count it taken when a slot holds it
        bool taken = inS(s, j);
        for (int i = 0; i < nn; ++i) taken |= add[i] == j;
        free_member = !taken;
      }
      if (!free_member) return false;
    }
    return true;
  }
  // Register slots take at most c - 3 of the chunk bits [0, c), so three lane
  // bits always remain inside the chunk; lane operations name up to 3 of them.
  bool tryAdd(StageBits& s, const SchedOp& op) const {
    if (s.dk) return false;
    if (op.k == 1) {
      const int b = op.q[0];
      const uint64_t bm = 1ULL << b;
      if (inS(s, b) || (s.lanereq & bm)) return true;
      if (b < c && __builtin_popcountll(s.lanereq) < kLaneBits && lowcount(s) <= c - kLaneBits) {
        s.lanereq |= bm;
        return true;
      }
      if (s.nS >= p.R) return false;
      if (b < c && lowcount(s) + 1 > c - kLaneBits) return false;
      s.S[s.nS++] = b;
      return true;
    }
    int need[2], nn = 0, lowadd = 0;
    for (int i = 0; i < 2; ++i)
      if (!inS(s, op.q[i])) { need[nn++] = op.q[i]; lowadd += op.q[i] < c; }
    if (s.nS + nn > p.R) return false;
    if (lowcount(s) + lowadd > lowlimit(s, op.grad != 0)) {
      // a stage without lane operations may hold more chunk bits as long as
      // its lanes can still be drawn with independent swizzle images; an empty
      // stage takes the operation regardless (its lanes may then share bank
      // groups: slower, still correct)
      if (s.lanereq != 0 || (s.nS > 0 && !lanes_feasible(s, need, nn))) return false;
    }
    for (int i = 0; i < nn; ++i) {
      s.S[s.nS++] = need[i];
      s.lanereq &= ~(1ULL << need[i]);   // earlier lane ops on this bit become slot ops
    }
    return true;
  }
  bool place(int idx, const SchedOp& op) {
    if (op.grad) {
      // adjoint steps want the psi / lambda select bit in register slot 0; slot
      // positions bind to operations only when the pass is finalised, so the
      // current stage can take the select bit into slot 0 (swapped there, or
      // inserted when a slot is free and the chunk-bit limit allows)
      if (!stages.empty() && !stages.back().dk) {
        StageBits trial = stages.back();
        const int sel = op.q[0];
        bool ready = trial.nS > 0 && trial.S[0] == sel;
        if (!ready && inS(trial, sel)) {
          for (int i = 1; i < trial.nS; ++i)
            if (trial.S[i] == sel) std::swap(trial.S[0], trial.S[i]);
          ready = true;
        } else if (!ready && trial.nS < p.R && !(trial.lanereq & (1ULL << sel)) &&
                   (sel >= c || lowcount(trial) + 1 <= lowlimit(trial, true))) {
          for (int i = trial.nS; i > 0; --i) trial.S[i] = trial.S[i - 1];
          trial.S[0] = sel;
          ++trial.nS;
          ready = true;
        }
        if (ready && tryAdd(trial, op)) {
          static_cast<StageBits&>(stages.back()) = trial;
          stages.back().ops.push_back(idx);
          return true;
        }
      }
      if ((int)stages.size() >= p.max_stages || (!allow_new && !stages.empty())) return false;
      Stage s;
      s.S[s.nS++] = op.q[0];
      if (!tryAdd(s, op)) return false;
      s.ops.push_back(idx);
      stages.push_back(std::move(s));
      return true;
    }
    if (op.k >= 3) {
      if (op.k > p.R) return false;
      if ((int)stages.size() >= p.max_stages || (!allow_new && !stages.empty())) return false;
      Stage s;
      s.dk = true;
      for (int i = 0; i < op.k; ++i) s.S[s.nS++] = op.q[i];
      s.ops.push_back(idx);
      stages.push_back(std::move(s));
      return true;
    }
    if (!stages.empty()) {
      StageBits trial = stages.back();
      if (tryAdd(trial, op)) {
        static_cast<StageBits&>(stages.back()) = trial;
        stages.back().ops.push_back(idx);
        return true;
      }
    }
    if ((int)stages.size() >= p.max_stages || (!allow_new && !stages.empty())) return false;
    Stage s;
    if (!tryAdd(s, op)) return false;
    s.ops.push_back(idx);
    stages.push_back(std::move(s));
    return true;
  }
};

// Rank over GF(2) of the low three bits of swz(1 << j) for the lane bits: the
// eight lanes of an octet hit distinct shared-memory bank groups iff it is 3.
int lane_rank(const int* l) {
  uint32_t v[3];
  for (int i = 0; i < 3; ++i) v[i] = swz(1u << l[i]) & 7u;
  int r = 0;
  for (int bit = 0; bit < 3; ++bit) {
    int piv = -1;
    for (int i = r; i < 3; ++i)
      if (v[i] & (1u << bit)) { piv = i; break; }
    if (piv < 0) continue;
    std::swap(v[r], v[piv]);
    for (int i = 0; i < 3; ++i)
      if (i != r && (v[i] & (1u << bit))) v[i] ^= v[r];
    ++r;
  }
  return r;
}

// Choose the 3 lane bits (tile-local) among `cand`, containing `req`, with the
// best bank-group rank (ties: lowest bits).
bool choose_lanes(const std::vector<int>& cand, uint32_t req, int out[3]) {
  int best = -1;
  const int n = (int)cand.size();
  for (int a = 0; a < n; ++a)
    for (int b = a + 1; b < n; ++b)
      for (int d = b + 1; d < n; ++d) {
        const int l[3] = {cand[a], cand[b], cand[d]};
        const uint32_t m = (1u << l[0]) | (1u << l[1]) | (1u << l[2]);
        if ((m & req) != req) continue;
        const int r = lane_rank(l);
        if (r > best) {
          best = r;
          out[0] = l[0]; out[1] = l[1]; out[2] = l[2];
          if (r == 3) return true;
        }
      }
  return best >= 0;
}

inline uint64_t opmask(const SchedOp& op) {
  uint64_t m = 0;
  for (int i = 0; i < op.k; ++i) m |= 1ULL << op.q[i];
  return m;
}

}  // namespace

int plan_passes(const SchedParams& p, const std::vector<SchedOp>& ops, std::vector<PassPlan>& out,
                std::string& err) {
  const int nb = p.nbits;
  const int nops = (int)ops.size();
  if (p.R < 3 || p.R > kMaxK) { err = "register slots must be 3, 4 or 5"; return -1; }
  if (nb < p.R + kLaneBits) { err = "array too small for the tile kernel"; return -1; }
  const int M = std::min(p.M, nb);
  const bool whole = nb <= p.M;         // the whole array is one tile
  const int c = whole ? std::min(p.c, M) : p.c;
  if (M < p.R + kLaneBits || M > kMaxTileBits) { err = "tile bits out of range"; return -1; }
  if (c < 3 || c > 7) { err = "chunk bits must be 3..7"; return -1; }
  // a tile moves in 2^(M - c - 2) box copies, one per lane of the CTA's first 128 threads
  if (!whole && M - c - 2 > 7) { err = "too many tile copies: raise the chunk bits or lower the tile bits"; return -1; }
  if (!whole && M - c < kMaxK) { err = "tile must hold the chunk plus 5 free bits"; return -1; }

  for (int i = 0; i < nops; ++i) {
    const SchedOp& o = ops[i];
    if (o.k < 1 || o.k > kMaxK) { err = "operation width out of range"; return -1; }
    for (int j = 0; j < o.k; ++j) {
      if (o.q[j] >= nb) { err = "operation bit out of range"; return -1; }
      for (int l = 0; l < j; ++l)
        if (o.q[l] == o.q[j]) { err = "repeated operation bit"; return -1; }
    }
    if (o.k > p.R) { err = "dense block wider than the register slots"; return -1; }
  }

  // per-bit queues of op indices (dependency order).  An adjoint step applies
  // the same 2x2 to the psi and lambda halves and never mixes them, so steps on
  // different qubits commute (their gradient terms too: Im<lambda|P_b|psi> does
  // not change when a unitary on another qubit acts on both halves); when no
  // other operation touches the select bit, adjoint steps are ordered by their
  // qubit bit only.
  std::vector<uint8_t> other_use(nb, 0);
  for (int i = 0; i < nops; ++i)
    if (!ops[i].grad)
      for (int j = 0; j < ops[i].k; ++j) other_use[ops[i].q[j]] = 1;
  auto dep_first = [&](int i) { return (ops[i].grad && !other_use[ops[i].q[0]]) ? 1 : 0; };
  auto ndeps = [&](int i) { return ops[i].k - dep_first(i); };
  std::vector<std::vector<int>> q(nb);
  std::vector<size_t> head(nb, 0);
  for (int i = 0; i < nops; ++i)
    for (int j = dep_first(i); j < ops[i].k; ++j) q[ops[i].q[j]].push_back(i);
  std::vector<int> headcnt(nops, 0);
  struct Facts { uint64_t mask; double cost; int elems; };   // looked up once per pass and operation below
  std::vector<Facts> facts(nops);
  for (int i = 0; i < nops; ++i) facts[i] = {opmask(ops[i]), op_cost(ops[i], p.grad_cost), op_mat_elems(ops[i])};
  std::set<int> ready;
  for (int b = 0; b < nb; ++b)
    if (!q[b].empty()) {
      int i = q[b][0];
      if (++headcnt[i] == ndeps(i)) ready.insert(i);
    }
  auto retire = [&](int i) {
    for (int j = dep_first(i); j < ops[i].k; ++j) {
      int b = ops[i].q[j];
      ++head[b];
      if (head[b] < q[b].size()) {
        int nx = q[b][head[b]];
        if (++headcnt[nx] == ndeps(nx)) ready.insert(nx);
      }
    }
  };

  const uint64_t lowmask = (c >= 64) ? ~0ULL : ((1ULL << c) - 1);
  const uint64_t allmask = (nb >= 64) ? ~0ULL : ((1ULL << nb) - 1);
  // the psi / lambda select bit of adjoint steps is local in every pass (as
  // the chunk bits are): otherwise passes widened by the fixed gates first
  // would leave it out and the steps could not join them
  uint64_t select_mask = 0;
  for (int i = 0; i < nops; ++i)
    if (ops[i].grad) select_mask |= 1ULL << ops[i].q[0];
  select_mask &= ~lowmask;
  int scheduled = 0;
  while (scheduled < nops) {
    if (ready.empty()) { err = "scheduler found no ready operation"; return -1; }
    uint64_t local = whole ? allmask : (lowmask | select_mask);
    int free_slots = whole ? 0 : (M - c - __builtin_popcountll(select_mask));
    PassBuilder pb(p, c);
    std::vector<int> taken;
    double cost = 0.0;
    int mat_elems = 0;
    int ngrad = 0;
    for (;;) {
      // every ready operation that fits the current stage joins it before an
      // operation may open the next stage
      bool progress = true;
      while (progress) {
        progress = false;
        for (int phase = 0; phase < 2 && !progress; ++phase) {
          pb.allow_new = phase == 1;
          for (auto it = ready.begin(); it != ready.end();) {
            const int i = *it;
            const SchedOp& o = ops[i];
            const double oc = facts[i].cost;
            if ((facts[i].mask & ~local) == 0 && (int)taken.size() < kMaxPassOps &&
                mat_elems + facts[i].elems <= kSmemMatElems && (taken.empty() || cost + oc <= p.budget) &&
                (!o.grad || ngrad < kMaxPassGrads) && pb.place(i, o)) {
              taken.push_back(i);
              cost += oc;
              mat_elems += facts[i].elems;
              ngrad += o.grad ? 1 : 0;
              it = ready.erase(it);
              retire(i);
              progress = true;
              if (phase == 1) break;   // one operation opens the stage; the others try to join it
            } else {
              ++it;
            }
          }
        }
      }
      pb.allow_new = true;
      if (free_slots == 0 || (int)taken.size() >= kMaxPassOps) break;
      int best = -1, bestmiss = 0;
      for (int i : ready) {
        const int miss = __builtin_popcountll(facts[i].mask & ~local);
        if (miss > 0 && miss <= free_slots && (taken.empty() || cost + facts[i].cost <= p.budget)) {
          best = i;
          bestmiss = miss;
          break;
        }
      }
      if (best < 0) break;
      local |= facts[best].mask;
      free_slots -= bestmiss;
    }
    if (taken.empty()) { err = "scheduler could not place an operation"; return -1; }
    scheduled += (int)taken.size();

    // ---- finalize: tile-local numbering, padded register slots, encoded ops
    PassPlan plan;
    std::memset(&plan.desc, 0, sizeof(plan.desc));
    PassDesc& d = plan.desc;
    std::vector<int> H;
    for (int b = c; b < nb; ++b)
      if (local & (1ULL << b)) H.push_back(b);
    for (int b = nb - 1; (int)H.size() < M - c && b >= c; --b)
      if (!(local & (1ULL << b))) H.push_back(b);
    std::sort(H.begin(), H.end());
    int pos[64];
    for (int b = 0; b < 64; ++b) pos[b] = -1;
    for (int b = 0; b < c; ++b) pos[b] = b;
    for (size_t i = 0; i < H.size(); ++i) pos[H[i]] = c + (int)i;
    d.M = (uint8_t)M;
    d.c = (uint8_t)c;
    d.R = (uint8_t)p.R;
    d.nH = (uint8_t)H.size();
    for (size_t i = 0; i < H.size(); ++i) d.H[i] = (uint8_t)H[i];
    // the copies' boxes span the first two runs of adjacent high bits (at most 256 entries per dimension)
    auto run = [&](size_t from) {
      size_t k = 0;
      while (from + k < H.size() && k < 8 && H[from + k] == H[from] + (int)k) ++k;
      return (int)k;
    };
    d.run1 = (uint8_t)run(0);
    d.nbox = (uint8_t)(d.run1 + run(d.run1));
    d.ntiles = 1ULL << (nb - M);
    d.nstages = (uint8_t)pb.stages.size();
    d.ngrad = 0;
    int nout = 0;
    for (size_t si = 0; si < pb.stages.size(); ++si) {
      const Stage& s = pb.stages[si];
      StageDesc& sd = d.st[si];
      bool used[kMaxTileBits] = {};
      int slot_of[kMaxTileBits];
      for (int j = 0; j < kMaxTileBits; ++j) slot_of[j] = -1;
      int nS = 0;
      for (int i = 0; i < s.nS; ++i) {
        const int j = pos[s.S[i]];
        sd.S[nS] = (uint8_t)j;
        slot_of[j] = nS++;
        used[j] = true;
      }
      // lanes: chunk bits for stages with lane operations, any tile bit for the
      // others; padding slots come from the highest bits left over
      uint32_t req = 0;
      for (int b = 0; b < c; ++b)
        if (s.lanereq & (1ULL << b)) req |= 1u << pos[b];
      std::vector<int> cand;
      const int lim = s.lanereq ? c : M;
      for (int j = 0; j < lim; ++j)
        if (!used[j]) cand.push_back(j);
      // keep R - nS bits for padding out of the candidates' reach when possible
      int lanes[3];
      if (!choose_lanes(cand, req, lanes)) { err = "internal: no lane bits for a stage"; return -1; }
      int lane_of[kMaxTileBits];
      for (int j = 0; j < kMaxTileBits; ++j) lane_of[j] = -1;
      for (int l = 0; l < kLaneBits; ++l) {
        sd.lane[l] = (uint8_t)lanes[l];
        lane_of[lanes[l]] = l;
        used[lanes[l]] = true;
      }
      for (int j = M - 1; nS < p.R && j >= 0; --j)
        if (!used[j]) { sd.S[nS] = (uint8_t)j; slot_of[j] = nS++; used[j] = true; }
      if (nS < p.R) { err = "internal: not enough tile bits for the register slots"; return -1; }
      sd.nt = 0;
      for (int j = 0; j < M; ++j)
        if (!used[j]) sd.tb[sd.nt++] = (uint8_t)j;
      sd.op0 = (uint16_t)nout;
      for (int i : s.ops) {
        const SchedOp& o = ops[i];
        plan.src.push_back((uint32_t)i);
        OpDesc& od = d.ops[nout++];
        od.k = o.k;
        od.mat = o.mat;
        od.perm = o.perm;
        od.flags = o.unit ? OPF_UNIT_PHASE : 0;
        od.urows = o.mono ? o.urows : 0;
        if (o.k == 1) {
          const int j = pos[o.q[0]];
          if (slot_of[j] >= 0) {
            od.kind = o.mono ? OP_M1R : (o.rot ? OP_R1R : (o.norm ? OP_N1R : OP_D1R));
            if (od.kind == OP_D1R && o.realm) od.flags |= OPF_REAL;
            od.a = (uint8_t)slot_of[j];
            if (o.norm) od.perm = (uint8_t)(o.norm - 1);
            if (o.rot) od.perm = (uint8_t)(o.rot - 1);
          }
          else if (lane_of[j] >= 0) {
            od.kind = o.mono ? OP_M1L : (o.rot ? OP_R1L : OP_D1L);
            if (od.kind == OP_D1L && o.realm && !o.norm) od.flags |= OPF_REAL;
            od.a = (uint8_t)lane_of[j];
            if (o.rot) od.perm = (uint8_t)(o.rot - 1);
          }
          else { err = "internal: 1q operation bit is neither a slot nor a lane"; return -1; }
        } else if (o.k == 2) {
          const int j0 = pos[o.q[0]], j1 = pos[o.q[1]];
          if (slot_of[j0] < 0 || slot_of[j1] < 0) { err = "internal: 2q operation outside slots"; return -1; }
          od.kind = o.grad ? OP_GRAD2 : (o.mono ? OP_M2R : (o.xpat ? OP_X2R : OP_D2R));
          if (od.kind == OP_X2R) od.flags = (uint8_t)(o.xpat >> 1);   // XPAT_* >> 1: bit 0 corners, bit 1 middle real
          od.a = (uint8_t)slot_of[j0];
          od.b = (uint8_t)slot_of[j1];
          if (o.grad) {
            od.perm = o.gen;
            od.flags = o.rot;                  // the inverse rotation's form (GradForm)
            od.gidx = d.ngrad;                 // local index; the global term goes to grad_term
            d.grad_term[d.ngrad++] = o.gidx;
          }
        } else {
          for (int t = 0; t < o.k; ++t)
            if (slot_of[pos[o.q[t]]] != t) { err = "internal: dense block slots out of order"; return -1; }
          od.kind = OP_DKR;
        }
      }
      sd.op1 = (uint16_t)nout;
    }
    d.nops = (uint32_t)nout;
    d.grad_base = 0;
    plan.nsrc = (int)taken.size();
    plan.cost = cost;
    out.push_back(std::move(plan));
  }
  return (int)out.size();
}

namespace {

using M4 = std::array<cplx64, 16>;

inline cplx64 cm(cplx64 a, cplx64 b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
inline cplx64 ca(cplx64 a, cplx64 b) { return {a.re + b.re, a.im + b.im}; }

M4 mul4(const M4& A, const M4& B) {
  M4 C;
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      cplx64 acc{0.0, 0.0};
      for (int k = 0; k < 4; ++k) acc = ca(acc, cm(A[r * 4 + k], B[k * 4 + c]));
      C[r * 4 + c] = acc;
    }
  return C;
}

// 2x2 U acting on local bit `bit` of a two-bit index (bit 0 = list[0])
M4 lift1(const cplx64* U, int bit) {
  M4 L;
  for (auto& x : L) x = {0.0, 0.0};
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      const int ob = bit ^ 1;
      if (((r >> ob) & 1) != ((c >> ob) & 1)) continue;
      L[r * 4 + c] = U[((r >> bit) & 1) * 2 + ((c >> bit) & 1)];
    }
  return L;
}

// 4x4 U on list (u0, u1) re-expressed on list (l0, l1) = (u1, u0)
M4 swap_bits(const cplx64* U) {
  M4 L;
  auto sw = [](int i) { return ((i & 1) << 1) | ((i >> 1) & 1); };
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) L[sw(r) * 4 + sw(c)] = U[r * 4 + c];
  return L;
}

struct Block {
  int k = 0;
  int q[2] = {-1, -1};
  M4 m;                 // dense (1q blocks use the top-left 2x2 in m[0], m[1], m[4], m[5])
  bool dead = false;
  int src = -1;         // index of the original op when the block is that op unchanged
  bool changed = false;
  bool xpat = false;    // a run of OP_X2R-shaped operations on one pair, kept apart from one-qubit blocks
};

// The phases at either end of a run of one-qubit operations between barriers (of
// which `ends` says where they are).  They stay out of the run's product: the
// decomposition carries them along as they are, where a product's entries would
// give them back up to rounding only, as phases that are 1 or not by the angles.
template <class Barrier>
std::vector<uint8_t> phases_at_ends(const std::vector<SchedOp>& ops, const std::vector<cplx64>& pool, Barrier ends) {
  struct Run { bool only = true, dense = false; std::vector<size_t> tail; };   // only: since a barrier, one-qubit operations
  std::vector<Run> runs(64);
  std::vector<uint8_t> alone(ops.size(), 0);
  auto unit = [](cplx64 a) { return std::fabs(a.re * a.re + a.im * a.im - 1.0) < 1e-12; };
  auto end = [&](Run& r) {
    if (r.only)
      for (size_t i : r.tail) alone[i] = 1;
    r = Run{};
  };
  for (size_t i = 0; i < ops.size(); ++i) {
    const SchedOp& o = ops[i];
    if (ends(o)) {
      for (int j = 0; j < o.k; ++j) end(runs[o.q[j]]);
    } else if (o.k == 2) {
      for (int j = 0; j < 2; ++j) {
        runs[o.q[j]].only = false;
        runs[o.q[j]].tail.clear();
      }
    } else {
      Run& r = runs[o.q[0]];
      if (!o.mono || (o.perm & 1) || (!o.unit && !(unit(pool[o.mat]) && unit(pool[o.mat + 1])))) {
        r.dense = true;
        r.tail.clear();
      } else if (r.only && !r.dense) {
        alone[i] = 1;
      } else {
        r.tail.push_back(i);
      }
    }
  }
  for (Run& r : runs) end(r);
  return alone;
}

}  // namespace

std::vector<SchedOp> fuse_two_qubit_blocks(const std::vector<SchedOp>& ops, std::vector<cplx64>& pool,
                                           bool monomial_barrier) {
  const int nb = 64;
  std::vector<Block> blocks;
  blocks.reserve(ops.size());
  std::vector<int> open(nb, -1), last(nb, -1);
  std::vector<int> passthrough;   // ops of width >= 3 keep their place as blocks with k = 0
  auto mat2 = [&](const SchedOp& o) {
    M4 m;
    const cplx64* U = pool.data() + o.dense;
    m[0] = U[0]; m[1] = U[1]; m[4] = U[2]; m[5] = U[3];
    return m;
  };
  std::vector<uint8_t> alone;
  if (monomial_barrier)
    alone = phases_at_ends(ops, pool, [](const SchedOp& o) {   // what ends a run in the loop below
      return o.k >= 3 || o.grad || o.smul != 0.0 || (o.k == 2 && (o.mono || o.xpat));
    });
  for (size_t i = 0; i < ops.size(); ++i) {
    const SchedOp& o = ops[i];
    // wide blocks and adjoint steps pass through unchanged, and so do two-qubit
    // monomials (CX, CZ, SWAP) when they are cheaper alone than inside a 4x4
    // adjoint steps and the scalars of a scaled backward sweep (smul) keep their place unchanged
    const bool diagonal2 = o.k == 2 && o.mono && o.perm == 0xE4;   // rows read their own column
    if (monomial_barrier && o.k == 2 && (o.xpat || diagonal2) && !o.grad && o.smul == 0.0) {
      // channel-shaped operations (OP_X2R's shape; diagonal ones included)
      // stay out of one-qubit blocks (a unitary inside would make the block
      // dense); consecutive ones on the same pair multiply into one block of
      // the same shape.  A run of one operation keeps it unchanged.
      const int a = o.q[0], bq = o.q[1];
      const int B = last[a];
      const cplx64* U = pool.data() + o.dense;
      M4 Um;
      for (int j = 0; j < 16; ++j) Um[j] = U[j];
      if (B >= 0 && B == last[bq] && blocks[B].xpat) {
        Block& bl = blocks[B];
        bl.m = mul4(bl.q[0] == a ? Um : swap_bits(Um.data()), bl.m);
        bl.changed = true;
        bl.src = -1;
        continue;
      }
      open[a] = open[bq] = -1;
      last[a] = last[bq] = (int)blocks.size();
      Block b;
      b.k = 2;
      b.q[0] = a;
      b.q[1] = bq;
      b.m = Um;
      b.src = (int)i;
      b.xpat = true;
      blocks.push_back(b);
      continue;
    }
    if (o.k >= 3 || o.grad || o.smul != 0.0 || (monomial_barrier && ((o.k == 2 && o.mono) || alone[i]))) {
      for (int j = 0; j < o.k; ++j) { open[o.q[j]] = -1; last[o.q[j]] = (int)blocks.size(); }
      Block b;
      b.k = 0;
      b.src = (int)i;
      blocks.push_back(b);
      continue;
    }
    if (o.k == 1) {
      const int a = o.q[0];
      const int B = open[a];
      if (B >= 0 && last[a] == B) {
        Block& bl = blocks[B];
        const cplx64 U[4] = {pool[o.dense], pool[o.dense + 1], pool[o.dense + 2], pool[o.dense + 3]};
        if (bl.k == 1) {
          M4 u1 = mat2(o);
          M4 r;
          for (auto& x : r) x = {0.0, 0.0};
          for (int rr = 0; rr < 2; ++rr)
            for (int cc = 0; cc < 2; ++cc)
              for (int kk = 0; kk < 2; ++kk)
                r[rr * 4 + cc] = ca(r[rr * 4 + cc], cm(u1[rr * 4 + kk], bl.m[kk * 4 + cc]));
          bl.m = r;
        } else {
          bl.m = mul4(lift1(U, bl.q[0] == a ? 0 : 1), bl.m);
        }
        bl.changed = true;
        bl.src = -1;
        continue;
      }
      Block b;
      b.k = 1;
      b.q[0] = a;
      b.m = mat2(o);
      b.src = (int)i;
      open[a] = last[a] = (int)blocks.size();
      blocks.push_back(b);
      continue;
    }
    // two-qubit op on list (a, b) (bit 0 = a)
    const int a = o.q[0], bq = o.q[1];
    const int Ba = open[a], Bb = open[bq];
    const cplx64* U = pool.data() + o.dense;
    M4 Um;
    for (int j = 0; j < 16; ++j) Um[j] = U[j];
    if (Ba >= 0 && Ba == Bb && last[a] == Ba && last[bq] == Ba && blocks[Ba].k == 2) {
      Block& bl = blocks[Ba];
      bl.m = mul4(bl.q[0] == a ? Um : swap_bits(Um.data()), bl.m);
      bl.changed = true;
      bl.src = -1;
      continue;
    }
    const bool okA = Ba < 0 || (blocks[Ba].k == 1 && last[a] == Ba);
    const bool okB = Bb < 0 || (blocks[Bb].k == 1 && last[bq] == Bb);
    const int posc = std::max(Ba, Bb);
    // the fused block goes to position posc: nothing after it may touch a or b
    const bool okPos = posc >= 0 && last[a] <= posc && last[bq] <= posc;
    Block nbk;
    nbk.k = 2;
    nbk.q[0] = a;
    nbk.q[1] = bq;
    if (okA && okB && okPos) {
      // the fused block sits at the later of the two one-qubit blocks; moving the
      // earlier one there is valid because it is the last block on its qubit
      M4 pre;
      for (auto& x : pre) x = {0.0, 0.0};
      for (int j = 0; j < 4; ++j) pre[j * 5] = {1.0, 0.0};
      if (Ba >= 0) {
        const cplx64 ua[4] = {blocks[Ba].m[0], blocks[Ba].m[1], blocks[Ba].m[4], blocks[Ba].m[5]};
        pre = mul4(lift1(ua, 0), pre);
      }
      if (Bb >= 0) {
        const cplx64 ub[4] = {blocks[Bb].m[0], blocks[Bb].m[1], blocks[Bb].m[4], blocks[Bb].m[5]};
        pre = mul4(lift1(ub, 1), pre);
      }
      nbk.m = mul4(Um, pre);
      nbk.changed = true;
      const int pos = std::max(Ba, Bb);
      const int other = std::min(Ba, Bb);
      if (other >= 0 && other != pos) blocks[other].dead = true;
      blocks[pos] = nbk;
      open[a] = open[bq] = last[a] = last[bq] = pos;
      continue;
    }
    nbk.m = Um;
    nbk.src = (int)i;
    open[a] = open[bq] = last[a] = last[bq] = (int)blocks.size();
    blocks.push_back(nbk);
  }
  std::vector<SchedOp> out;
  out.reserve(blocks.size());
  for (const Block& b : blocks) {
    if (b.dead) continue;
    if (b.src >= 0 && !b.changed) {
      out.push_back(ops[b.src]);
      continue;
    }
    SchedOp o{};
    o.k = (uint8_t)b.k;
    const int d = 1 << b.k;
    o.dense = (uint32_t)pool.size();
    double flat[32];
    for (int r = 0; r < d; ++r)
      for (int c = 0; c < d; ++c) {
        const cplx64 v = b.m[r * 4 + c];
        pool.push_back(v);
        flat[2 * (r * d + c)] = v.re;
        flat[2 * (r * d + c) + 1] = v.im;
      }
    for (int j = 0; j < b.k; ++j) o.q[j] = (uint8_t)b.q[j];
    o.mat = o.dense;
    double ph[8];
    uint8_t perm = 0, unit = 0;
    if (classify_monomial(flat, b.k, &perm, ph, &unit)) {
      o.mono = 1;
      o.perm = perm;
      o.unit = unit;
      o.mat = (uint32_t)pool.size();
      for (int j = 0; j < d; ++j) pool.push_back({ph[2 * j], ph[2 * j + 1]});
    } else if (b.k == 2) {
      o.xpat = (uint8_t)classify_xpattern(flat);
    }
    out.push_back(o);
  }
  return out;
}

void normalize_one_qubit_ops(std::vector<SchedOp>& ops, std::vector<cplx64>& pool) {
  std::vector<int> dense1;
  for (size_t i = 0; i < ops.size(); ++i)
    if (ops[i].k == 1 && !ops[i].mono && !ops[i].grad && !ops[i].rot && !ops[i].realm) dense1.push_back((int)i);
  for (size_t s0 = 0; s0 < dense1.size(); s0 += kNormSegment) {
    const size_t s1 = std::min(dense1.size(), s0 + kNormSegment);
    if (s1 - s0 < 2) break;
    cplx64 scale{1.0, 0.0};
    for (size_t j = s0; j + 1 < s1; ++j) {
      SchedOp& o = ops[dense1[j]];
      const cplx64* U = pool.data() + o.dense;
      const int col = (std::hypot(U[1].re, U[1].im) > std::hypot(U[0].re, U[0].im)) ? 1 : 0;
      const cplx64 s = U[col];
      const double n2 = s.re * s.re + s.im * s.im;
      const cplx64 inv{s.re / n2, -s.im / n2};
      const uint32_t at = (uint32_t)pool.size();
      for (int e = 0; e < 4; ++e) pool.push_back(e == col ? cplx64{1.0, 0.0} : cm(pool[o.dense + e], inv));
      o.dense = o.mat = at;
      o.norm = (uint8_t)(col + 1);
      o.realm = 0;
      scale = cm(scale, s);
    }
    SchedOp& c = ops[dense1[s1 - 1]];   // the run's carrier takes the product of the divisors
    const uint32_t at = (uint32_t)pool.size();
    for (int e = 0; e < 4; ++e) pool.push_back(cm(pool[c.dense + e], scale));
    c.dense = c.mat = at;
    c.realm = 0;
  }
}

namespace {

// A product or quotient in extended precision, rounded once: the scalar of a
// whole circuit, the entries of merged diagonals, phases.  (|b|^2 of a phase
// rounded to double before a division is biased: the grid is twice as coarse
// above 1 as below.)
struct WideScalar {
  long double re = 1.0L, im = 0.0L;
  void times(WideScalar f) {
    const long double r = re * f.re - im * f.im;
    im = re * f.im + im * f.re;
    re = r;
  }
  void times(cplx64 f) { times(WideScalar{f.re, f.im}); }
  WideScalar inverse() const {
    const long double n = re * re + im * im;
    return {re / n, -im / n};
  }
  cplx64 rounded() const { return {(double)re, (double)im}; }
};
WideScalar quotient(cplx64 a, cplx64 b) {
  const long double n = (long double)b.re * b.re + (long double)b.im * b.im;
  return {((long double)a.re * b.re + (long double)a.im * b.im) / n, ((long double)a.im * b.re - (long double)a.re * b.im) / n};
}
inline cplx64 cdiv(cplx64 a, cplx64 b) { return quotient(a, b).rounded(); }
inline double cabs2(cplx64 a) { return a.re * a.re + a.im * a.im; }
inline bool is_one(cplx64 a) { return a.re == 1.0 && a.im == 0.0; }

// A phase is dropped only where it is exactly 1.  So that an operation does not
// come and go with the rounding of the angles, phases that cancel come out
// exactly 1: a pending diagonal is kept as diag(1, b), the phases of a gate's
// entries are taken relative to its own first entry, and what does not enter a
// phase is not multiplied into it; where rounding decides (a product of complex
// gates), the phase is emitted even if it is 1 (dense1).
struct Decomposer {
  std::vector<SchedOp>& out;
  std::vector<cplx64>& pool;
  std::vector<cplx64> pa, pb;   // pending output diagonal diag(pa[q], pb[q]) of each qubit (set_pending)
  std::vector<uint8_t> px;      // a pending X of the qubit, before that diagonal (modes that carry them)
  // DECOMP_STEADY_ENDS: the angles decide whether an X (bit 0) or a sign of the
  // pending diagonal (bit 1) is pending
  std::vector<uint8_t> open;
  WideScalar G;                 // scalar factored out of the emitted operations
  DecompMode mode;
  int rotations = 0;            // since the last scalar
  // a tan form divides by c >= 1/sqrt 2: this many keep the scale above 2^-96
  static constexpr int kScalarEvery = 192;

  Decomposer(std::vector<SchedOp>& o, std::vector<cplx64>& p, DecompMode m)
      : out(o), pool(p), pa(64, {1.0, 0.0}), pb(64, {1.0, 0.0}), px(64, 0), open(64, 0), mode(m) {}
  bool carries() const { return mode == DECOMP_STEADY || mode == DECOMP_STEADY_ENDS; }   // pending X operators

  // the pending diagonal of q becomes diag(a, b): diag(1, b / a), a in G, when
  // a has modulus 1 (other diagonals keep their scale to themselves)
  void set_pending(int q, cplx64 a, cplx64 b) {
    if (std::fabs(cabs2(a) - 1.0) < 1e-12 && !is_one(a)) {
      G.times(a);
      b = (b.re == a.re && b.im == a.im) ? cplx64{1.0, 0.0} : cdiv(b, a);
      a = {1.0, 0.0};
    }
    pa[q] = a;
    pb[q] = b;
  }
  uint32_t put(std::initializer_list<cplx64> v) {
    const uint32_t at = (uint32_t)pool.size();
    for (const cplx64& x : v) pool.push_back(x);
    return at;
  }
  // one-qubit diagonal diag(a, b) = a diag(1, b / a): the scalar goes to G
  void emit_phase(int q, cplx64 a, cplx64 b, bool always = false) {
    const cplx64 r = cdiv(b, a);
    G.times(a);
    if (is_one(r) && !always) return;
    SchedOp o{};
    o.k = 1;
    o.q[0] = (uint8_t)q;
    o.mono = 1;
    o.perm = 0;
    o.urows = 1;
    o.mat = put({{1.0, 0.0}, r});
    o.dense = put({{1.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, r});
    out.push_back(o);
  }
  void flush_x(int q) {
    if (!px[q]) return;
    emit_x(q);
    px[q] = 0;
  }
  void flush(int q) {
    flush_x(q);
    if (is_one(pa[q]) && is_one(pb[q])) return;
    emit_phase(q, pa[q], pb[q]);
    pa[q] = pb[q] = {1.0, 0.0};
  }
  // at the end of the list
  void close(int q) {
    if (mode == DECOMP_STEADY_ENDS && open[q]) {
      if (open[q] & 1) {   // X or the identity, as a real 2x2
        const cplx64 x{(double)px[q], 0.0}, i{1.0 - px[q], 0.0};
        SchedOp o{};
        o.k = 1;
        o.q[0] = (uint8_t)q;
        o.realm = 1;
        o.dense = o.mat = put({i, x, x, i});
        out.push_back(o);
        px[q] = 0;
      }
      emit_phase(q, pa[q], pb[q], true);
      pa[q] = pb[q] = {1.0, 0.0};
      return;
    }
    flush(q);
  }
  void emit_scalar(int q) {
    const cplx64 g = G.rounded();
    if (is_one(g)) return;
    SchedOp o{};
    o.k = 1;
    o.q[0] = (uint8_t)q;
    o.mono = 1;
    o.perm = 0;
    o.mat = put({g, g});
    o.dense = put({g, {0.0, 0.0}, {0.0, 0.0}, g});
    out.push_back(o);
    G = WideScalar{};
  }
  void emit_x(int q) {
    SchedOp o{};
    o.k = 1;
    o.q[0] = (uint8_t)q;
    o.mono = 1;
    o.perm = 1;
    o.unit = 1;
    o.urows = 3;
    o.mat = put({{1.0, 0.0}, {1.0, 0.0}});
    o.dense = put({{0.0, 0.0}, {1.0, 0.0}, {1.0, 0.0}, {0.0, 0.0}});
    out.push_back(o);
  }
  // [[c, -s], [s, c]] (c > 0) times the scalar g, normalised by max(c, |s|)
  void emit_rotation(int q, double c, double s, cplx64 g) {
    SchedOp o{};
    o.k = 1;
    o.q[0] = (uint8_t)q;
    if (c >= std::fabs(s)) {
      const double t = s / c;
      G.times(g);
      G.times(cplx64{c, 0.0});
      o.rot = 1;
      o.dense = put({{1.0, 0.0}, {-t, 0.0}, {t, 0.0}, {1.0, 0.0}});
    } else {
      const double u = c / s;
      G.times(g);
      G.times(cplx64{s, 0.0});
      o.rot = 2;
      o.dense = put({{u, 0.0}, {-1.0, 0.0}, {1.0, 0.0}, {u, 0.0}});
    }
    o.mat = o.dense;
    out.push_back(o);
    // keep the scale of the intermediate state within 2^+-100
    const double g2 = cabs2(G.rounded());
    ++rotations;
    if (g2 < 0x1p-200 || g2 > 0x1p200 || (mode != DECOMP_BY_ANGLE && rotations >= kScalarEvery)) {
      emit_scalar(q);
      rotations = 0;
    }
  }
  void emit_real(int q, double c, double s, cplx64 g) {   // [[c, -s], [s, c]] as it is, times g
    SchedOp o{};
    o.k = 1;
    o.q[0] = (uint8_t)q;
    o.realm = 1;
    o.dense = o.mat = put({{c, 0.0}, {-s, 0.0}, {s, 0.0}, {c, 0.0}});
    out.push_back(o);
    G.times(g);
  }
  // dense one-qubit U (row-major) on q, after the pending diagonal of q
  // (`last`: no dense one-qubit operation on q follows)
  void dense1(const SchedOp& src, bool last) {
    const int q = src.q[0];
    const bool steady = carries();
    const cplx64* U = pool.data() + src.dense;
    cplx64 A = U[0], B = U[1], C = U[2], D = U[3];
    if (px[q]) {   // the pending X swaps the columns, and the diagonal's entries with them
      std::swap(A, B);
      std::swap(C, D);
      set_pending(q, pb[q], pa[q]);
      px[q] = 0;
    }
    A = cm(A, pa[q]);
    B = cm(B, pb[q]);
    C = cm(C, pa[q]);
    D = cm(D, pb[q]);
    const double n0 = cabs2(A) + cabs2(C), n1 = cabs2(B) + cabs2(D);
    const cplx64 ip{A.re * B.re + A.im * B.im + C.re * D.re + C.im * D.im,
                    A.re * B.im - A.im * B.re + C.re * D.im - C.im * D.re};   // conj(A) B + conj(C) D
    const bool unitary = std::fabs(n0 - 1.0) < 1e-12 && std::fabs(n1 - 1.0) < 1e-12 && cabs2(ip) < 1e-24;
    const double c0 = std::sqrt(cabs2(A)), s0 = std::sqrt(cabs2(C));
    if (unitary && s0 == 0.0 && cabs2(B) == 0.0) {     // diagonal: joins the pending diagonal
      set_pending(q, A, D);
      return;
    }
    if (unitary && c0 == 0.0 && cabs2(D) == 0.0) {     // anti-diagonal: X, then diag(B, C)
      if (steady) px[q] = 1;
      else emit_x(q);
      set_pending(q, B, C);
      return;
    }
    if (unitary && c0 > 0.0 && s0 > 0.0) {
      // steady: U = X (X U) where |c| < |s|, so the rotation is always of the tan form
      const bool swap = steady && !last && c0 < s0;
      if (swap) {
        std::swap(A, C);
        std::swap(B, D);
      }
      // u diag(1, d) [[c, -s], [s, c]] diag(1, e), u the phase of A: a real gate gives d and e of exactly +-1
      const double c = swap ? s0 : c0;
      double s = swap ? c0 : s0;
      const cplx64 u{A.re / c, A.im / c};
      const cplx64 du = cdiv(C, u), eu = cdiv(B, u);   // divided: |u| is 1 up to rounding only, and the same way each time
      cplx64 d{du.re / s, du.im / s}, e{-eu.re / s, -eu.im / s};
      // A and B both real or both imaginary: e is 1 or not for every angle
      const bool exact = (A.im == 0.0 && B.im == 0.0) || (A.re == 0.0 && B.re == 0.0);
      // the sign goes to s: a real gate has no phase, whatever its angle (behind a pending one, none after it)
      if (mode != DECOMP_BY_ANGLE && (exact ? e.re < 0.0 : d.im == 0.0 && d.re < 0.0)) {
        s = -s;
        d = {-d.re, -d.im};
        e = {-e.re, -e.im};
      }
      const cplx64 Dr = cm(cm(u, cm(d, e)), {c, 0.0});      // the rebuilt entry D
      if (cabs2({Dr.re - D.re, Dr.im - D.im}) < 1e-28) {
        emit_phase(q, {1.0, 0.0}, e, mode != DECOMP_BY_ANGLE && !exact);
        if (steady && last) emit_real(q, c, s, u);
        else emit_rotation(q, c, s, u);
        px[q] = swap ? 1 : 0;
        open[q] = last ? (open[q] ? 2 : 0) : 3;
        set_pending(q, swap ? d : cplx64{1.0, 0.0}, swap ? cplx64{1.0, 0.0} : d);
        return;
      }
      if (swap) {
        std::swap(A, C);
        std::swap(B, D);
      }
    }
    // not unitary (or not rebuilt exactly enough): dense, with the pending diagonal in its columns
    SchedOp o = src;
    o.dense = o.mat = put({A, B, C, D});
    o.norm = 0;
    o.rot = 0;
    o.realm = 0;
    pa[q] = pb[q] = {1.0, 0.0};
    out.push_back(o);
  }
  // two-qubit monomial: the pending diagonals pass through the permutation and
  // factor per qubit; the non-factoring part is a phase on the |11> row
  void mono2(const SchedOp& src) {
    const int q0 = src.q[0], q1 = src.q[1];
    cplx64 ph[4];
    for (int r = 0; r < 4; ++r) ph[r] = src.unit ? cplx64{1.0, 0.0} : pool[src.mat + r];
    // pending X operators X^m in front of the permutation P are X^mo behind it
    // (every permutation of four is affine: P(r ^ mo) = P(r) ^ m); rows are
    // numbered before X^mo
    auto column = [&](int r) { return (src.perm >> (2 * r)) & 3; };
    const int m = (px[q0] ? 1 : 0) | (px[q1] ? 2 : 0);
    int mo = 0;
    while ((column(mo) ^ column(0)) != m) ++mo;
    if (open[q0] | open[q1]) {   // an X spreads as this permutation's does, its sign to both qubits
      int may = 0;
      for (int z = 1; z < 4; ++z)
        if (((column(z) ^ column(0)) & ~((open[q0] & 1) | (open[q1] & 1) << 1)) == 0) may |= z;
      open[q0] = (uint8_t)((may & 1) | 2);
      open[q1] = (uint8_t)((may >> 1) | 2);
    }
    cplx64 Dp[4], php[4];
    for (int z = 0; z < 4; ++z) {
      const int r = z ^ mo, col = column(r);
      const cplx64 dl = cm((col & 1) ? pb[q0] : pa[q0], (col & 2) ? pb[q1] : pa[q1]);
      Dp[z] = cm(ph[r], dl);
      php[z] = ph[r];
    }
    bool unit_modulus = true;
    for (int r = 0; r < 4; ++r) unit_modulus = unit_modulus && std::fabs(cabs2(ph[r]) - 1.0) < 1e-12;
    if (!unit_modulus) {
      // a non-unitary diagonal part (a channel's damping factors): carried on it
      // would make the next gates on these qubits non-unitary, so it keeps its
      // place with the pending diagonals folded into its phases
      SchedOp o = src;
      o.unit = 0;
      o.urows = 0;
      o.nrows = 0;
      px[q0] = (uint8_t)(mo & 1);
      px[q1] = (uint8_t)(mo >> 1);
      o.mat = put({Dp[0], Dp[1], Dp[2], Dp[3]});
      o.dense = (uint32_t)pool.size();
      for (int r = 0; r < 4; ++r)
        for (int c = 0; c < 4; ++c)
          pool.push_back(((src.perm >> (2 * r)) & 3) == c ? Dp[r] : cplx64{0.0, 0.0});
      pa[q0] = pa[q1] = pb[q0] = pb[q1] = {1.0, 0.0};
      out.push_back(o);
      return;
    }
    // Dp[z] = s0 x1^z0 y1^z1 gamma^(z0 z1): the gate's own phases, and of each
    // pending diag(a, b) the a in s0 and b / a by the bit of its qubit that row z
    // reads, an affine function of z0 and z1
    WideScalar s0, x1 = quotient(php[1], php[0]), y1 = quotient(php[2], php[0]), gamma = quotient(php[3], php[0]);
    s0.times(php[0]);
    gamma.times(x1.inverse());
    gamma.times(y1.inverse());
    for (int j = 0; j < 2; ++j) {
      const cplx64 a = pa[j ? q1 : q0];
      const WideScalar w = quotient(pb[j ? q1 : q0], a), wi = w.inverse();
      int bit[4];
      for (int z = 0; z < 4; ++z) bit[z] = (column(z ^ mo) >> j) & 1;
      s0.times(a);
      if (bit[0]) s0.times(w);
      if (bit[1] != bit[0]) x1.times(bit[1] ? w : wi);
      if (bit[2] != bit[0]) y1.times(bit[2] ? w : wi);
      for (int g = bit[3] + bit[0] - bit[1] - bit[2]; g; g += g > 0 ? -1 : 1) gamma.times(g > 0 ? w : wi);   // 0, 2 or -2
    }
    G.times(s0);
    px[q0] = (uint8_t)(mo & 1);
    px[q1] = (uint8_t)(mo >> 1);
    // the diagonal comes after the X
    const cplx64 one{1.0, 0.0}, xr = x1.rounded(), yr = y1.rounded(), gr = gamma.rounded();
    set_pending(q0, px[q0] ? xr : one, px[q0] ? one : xr);
    set_pending(q1, px[q1] ? yr : one, px[q1] ? one : yr);
    SchedOp o = src;
    const bool unit = is_one(gr);
    o.unit = unit ? 1 : 0;
    o.urows = unit ? 15 : 7;
    o.nrows = (gr.re == -1.0 && gr.im == 0.0) ? 8 : 0;
    o.mat = put({{1.0, 0.0}, {1.0, 0.0}, {1.0, 0.0}, gr});
    o.dense = (uint32_t)pool.size();
    for (int r = 0; r < 4; ++r)
      for (int c = 0; c < 4; ++c) {
        const bool hit = ((src.perm >> (2 * r)) & 3) == c;
        pool.push_back(hit ? (r == 3 ? gr : cplx64{1.0, 0.0}) : cplx64{0.0, 0.0});
      }
    out.push_back(o);
  }
  // dense k-qubit operation: the pending diagonals scale its columns
  // (and a pending X swaps them)
  void dense_k(const SchedOp& src) {
    const int d = 1 << src.k;
    int m = 0, keep = 0;
    for (int j = 0; j < src.k; ++j) m |= px[src.q[j]] ? 1 << j : 0;
    if (src.xpat && m) {
      // a channel's shape survives X (x) X on both sides only: those stay pending behind it
      if (m == 3) keep = 3;
      else for (int j = 0; j < src.k; ++j) flush_x(src.q[j]);
      if (m != 3) m = 0;
    }
    SchedOp o = src;
    o.dense = o.mat = (uint32_t)pool.size();
    // column c of the operation acting on X^m x reads column c ^ m, scaled by the diagonal there; rows
    // keep their X^keep in front
    for (int r = 0; r < d; ++r)
      for (int c = 0; c < d; ++c) {
        const int col = c ^ m;
        cplx64 f{1.0, 0.0};
        for (int j = 0; j < src.k; ++j) f = cm(f, ((col >> j) & 1) ? pb[src.q[j]] : pa[src.q[j]]);
        pool.push_back(cm(pool[src.dense + (r ^ keep) * d + col], f));
      }
    for (int j = 0; j < src.k; ++j) {
      pa[src.q[j]] = pb[src.q[j]] = {1.0, 0.0};
      px[src.q[j]] = (uint8_t)((keep >> j) & 1);
    }
    if (src.xpat)   // the diagonal scales columns: same shape, entries maybe complex now
      o.xpat = (uint8_t)classify_xpattern(reinterpret_cast<const double*>(pool.data() + o.dense));
    out.push_back(o);
  }
};

}  // namespace

void decompose_one_qubit_ops(std::vector<SchedOp>& ops, std::vector<cplx64>& pool, DecompMode mode) {
  std::vector<SchedOp> out;
  out.reserve(ops.size() * 2);
  Decomposer dc(out, pool, mode);
  std::vector<size_t> last(64, 0);   // index past each qubit's last dense one-qubit operation
  for (size_t i = 0; i < ops.size(); ++i)
    if (ops[i].k == 1 && !ops[i].mono && !ops[i].grad) last[ops[i].q[0]] = i + 1;
  int last_q = 0;
  for (size_t i = 0; i < ops.size(); ++i) {
    const SchedOp& o = ops[i];
    if (o.grad) {
      for (int j = 0; j < o.k; ++j) dc.flush(o.q[j]);
      out.push_back(o);
    } else if (o.k == 1 && !o.mono) {
      dc.dense1(o, last[o.q[0]] == i + 1);
    } else if (o.k == 1) {             // one-qubit monomial: diagonal, or X with phases
      const int q = o.q[0];
      const cplx64 p0 = o.unit ? cplx64{1.0, 0.0} : pool[o.mat], p1 = o.unit ? cplx64{1.0, 0.0} : pool[o.mat + 1];
      if (o.perm & 1) {
        if (dc.carries()) dc.px[q] ^= 1;
        else dc.emit_x(q);
        dc.set_pending(q, cm(p0, dc.pb[q]), cm(p1, dc.pa[q]));
      } else {
        dc.set_pending(q, cm(dc.pa[q], p0), cm(dc.pb[q], p1));
      }
    } else if (o.k == 2 && o.mono) {
      dc.mono2(o);
    } else {
      dc.dense_k(o);
    }
    last_q = o.q[0];
  }
  for (int q = 0; q < 64; ++q) dc.close(q);
  dc.emit_scalar(last_q);
  ops.swap(out);
}

// ------------------------------------------------------------ adjoint builder
namespace {

using cdd = std::complex<double>;

void push_op(std::vector<SchedOp>& out, std::vector<cplx64>& pool, int k, const int* q, const cdd* m) {
  SchedOp o{};
  o.k = (uint8_t)k;
  for (int i = 0; i < k; ++i) o.q[i] = (uint8_t)q[i];
  const int d = 1 << k;
  o.dense = o.mat = (uint32_t)pool.size();
  double flat[32];
  for (int i = 0; i < d * d; ++i) {
    pool.push_back({m[i].real(), m[i].imag()});
    flat[2 * i] = m[i].real();
    flat[2 * i + 1] = m[i].imag();
  }
  double ph[8];
  uint8_t perm = 0, unit = 0;
  if (classify_monomial(flat, k, &perm, ph, &unit)) {
    o.mono = 1;
    o.perm = perm;
    o.unit = unit;
    o.mat = (uint32_t)pool.size();
    for (int i = 0; i < d; ++i) {
      pool.push_back({ph[2 * i], ph[2 * i + 1]});
      if (ph[2 * i] == 1.0 && ph[2 * i + 1] == 0.0) o.urows |= (uint8_t)(1u << i);   // its product is skipped
      if (k == 2 && ph[2 * i] == -1.0 && ph[2 * i + 1] == 0.0) o.nrows |= (uint8_t)(1u << i);   // CZ
    }
  } else if (k == 1) {
    bool real = true;
    for (int i = 0; i < 4; ++i) real = real && flat[2 * i + 1] == 0.0;
    o.realm = real ? 1 : 0;
  }
  out.push_back(o);
}

// exp(-i theta P / 2) for P = X (g 0), Y (1), Z (2)
void rotation(int g, double th, cdd* m) {
  const double c = std::cos(th / 2.0), s = std::sin(th / 2.0);
  const cdd I(0.0, 1.0);
  if (g == 0) { m[0] = c; m[1] = -I * s; m[2] = -I * s; m[3] = c; }
  else if (g == 1) { m[0] = c; m[1] = -s; m[2] = s; m[3] = c; }
  else { m[0] = std::exp(-I * (th / 2.0)); m[1] = 0.0; m[2] = 0.0; m[3] = std::exp(I * (th / 2.0)); }
}

// the same from c = cos(th/2), s = sin(th/2)
void rotation_cs(int g, double c, double s, cdd* m) {
  const cdd I(0.0, 1.0);
  if (g == 0) { m[0] = c; m[1] = -I * s; m[2] = -I * s; m[3] = c; }
  else if (g == 1) { m[0] = c; m[1] = -s; m[2] = s; m[3] = c; }
  else { m[0] = cdd(c, -s); m[1] = 0.0; m[2] = 0.0; m[3] = cdd(c, s); }
}

void dagger2(const cdd* m, cdd* o) {
  o[0] = std::conj(m[0]); o[1] = std::conj(m[2]); o[2] = std::conj(m[1]); o[3] = std::conj(m[3]);
}

// the rotations a parametrised gate is made of, in forward order: (generator, parameter)
int rotations_of(const AnsatzOp& op, int gen[3], int par[3]) {
  switch (op.kind) {
    case GATE_RX: gen[0] = 0; par[0] = op.param; return 1;
    case GATE_RY: gen[0] = 1; par[0] = op.param; return 1;
    case GATE_RZ: case GATE_P: gen[0] = 2; par[0] = op.param; return 1;
    // U3(theta, phi, lambda) = e^{i (phi + lambda) / 2} Rz(phi) Ry(theta) Rz(lambda)
    case GATE_U3: gen[0] = 2; par[0] = op.param + 2; gen[1] = 1; par[1] = op.param; gen[2] = 2; par[2] = op.param + 1;
      return 3;
    default: return 0;
  }
}

void fixed_matrix(const AnsatzOp& op, int& k, int q[2], cdd* m) {
  const double r = 1.0 / std::sqrt(2.0);
  const cdd I(0.0, 1.0);
  for (int i = 0; i < 16; ++i) m[i] = 0.0;
  switch (op.kind) {
    case GATE_H: k = 1; q[0] = op.q0; m[0] = r; m[1] = r; m[2] = r; m[3] = -r; return;
    case GATE_X: k = 1; q[0] = op.q0; m[1] = 1.0; m[2] = 1.0; return;
    case GATE_SX: k = 1; q[0] = op.q0; m[0] = 0.5 * (1.0 + I); m[1] = 0.5 * (1.0 - I); m[2] = 0.5 * (1.0 - I);
      m[3] = 0.5 * (1.0 + I); return;
    case GATE_CZ: k = 2; q[0] = op.q1; q[1] = op.q0; m[0] = 1.0; m[5] = 1.0; m[10] = 1.0; m[15] = -1.0; return;
    case GATE_CX:   // local bit 1 = control q0, bit 0 = target q1
      k = 2; q[0] = op.q1; q[1] = op.q0; m[0] = 1.0; m[5] = 1.0; m[11] = 1.0; m[14] = 1.0; return;
    default: k = 0; return;
  }
}

}  // namespace

int ansatz_check(int n, const std::vector<AnsatzOp>& ops, std::string& err) {
  int np = 0;
  for (const AnsatzOp& o : ops) {
    if (o.kind < GATE_RX || o.kind > GATE_SX) { err = "unknown gate kind"; return -1; }
    if (o.q0 < 0 || o.q0 >= n) { err = "qubit out of range"; return -1; }
    if (o.kind == GATE_CZ || o.kind == GATE_CX) {
      if (o.q1 < 0 || o.q1 >= n || o.q1 == o.q0) { err = "invalid second qubit"; return -1; }
    }
    if (o.kind <= GATE_P) {
      if (o.param < 0) { err = "parametrised gate without a parameter index"; return -1; }
      np = std::max(np, o.param + (o.kind == GATE_U3 ? 3 : 1));
    }
  }
  return np;
}

void pauli_frame(const std::vector<AnsatzOp>& ops, const double* params, PauliFrame& f) {
  f.rot.clear();
  f.x = f.z = 0;
  for (const AnsatzOp& o : ops) {
    int gen[3], par[3];
    const int nr = rotations_of(o, gen, par);
    const uint64_t b = 1ULL << o.q0;
    for (int r = 0; r < nr; ++r) {
      const bool fx = f.x & b, fz = f.z & b;
      // X, Y, Z anticommute with the frame's Pauli operator on the qubit
      const bool anti = gen[r] == 0 ? fz : (gen[r] == 1 ? fx != fz : fx);
      PauliFrame::Rot t;
      t.sign = anti ? -1 : 1;
      const double th = params[par[r]];
      t.c = std::cos(th / 2.0);
      t.s = t.sign * std::sin(th / 2.0);
      if (gen[r] != 2 && std::fabs(t.s) > std::fabs(t.c)) {
        // th' = th - pi: cos(th'/2) = sin(th/2), sin(th'/2) = -cos(th/2); exp(-i pi P / 2) joins the frame
        const double c = t.c;
        t.c = t.s;
        t.s = -c;
        f.x ^= b;
        if (gen[r] == 1) f.z ^= b;
      }
      if (gen[r] != 2 && t.c < 0.0) {   // an overall sign
        t.c = -t.c;
        t.s = -t.s;
      }
      f.rot.push_back(t);
    }
    if (nr) continue;
    const uint64_t c = o.q1 >= 0 ? 1ULL << o.q1 : 0;
    switch (o.kind) {
      case GATE_CZ:
        if (f.x & b) f.z ^= c;
        if (f.x & c) f.z ^= b;
        break;
      case GATE_CX:   // control q0, target q1
        if (f.x & b) f.x ^= c;
        if (f.z & c) f.z ^= b;
        break;
      case GATE_H: {
        const bool fx = f.x & b, fz = f.z & b;
        f.x = (f.x & ~b) | (fz ? b : 0);
        f.z = (f.z & ~b) | (fx ? b : 0);
        break;
      }
      case GATE_SX:   // Z to -Y
        if (f.z & b) f.x ^= b;
        break;
      default: break;
    }
  }
}

void ansatz_forward(int n, const std::vector<AnsatzOp>& ops, const double* params, std::vector<SchedOp>& out,
                    std::vector<cplx64>& pool, bool phase_free, const PauliFrame* frame) {
  (void)n;
  size_t rot = 0;
  for (const AnsatzOp& o : ops) {
    int gen[3], par[3];
    const int nr = rotations_of(o, gen, par);
    if (nr) {
      for (int r = 0; r < nr; ++r) {
        cdd m[4];
        if (frame) rotation_cs(gen[r], frame->rot[rot].c, frame->rot[rot].s, m);
        else rotation(gen[r], params[par[r]], m);
        if (phase_free && gen[r] == 2) {   // e^{-i th/2} diag(1, e^{i th}): the common phase dropped
          const double th = params[par[r]];
          m[0] = 1.0;
          m[3] = cdd(std::cos(th), frame ? frame->rot[rot].sign * std::sin(th) : std::sin(th));
        }
        ++rot;
        const int q[1] = {o.q0};
        push_op(out, pool, 1, q, m);
      }
      continue;
    }
    int k, q[2];
    cdd m[16];
    fixed_matrix(o, k, q, m);
    push_op(out, pool, k, q, m);
  }
}

void ansatz_backward(int n, const std::vector<AnsatzOp>& ops, const double* params, std::vector<SchedOp>& out,
                     std::vector<cplx64>& pool, std::vector<int>& grad_param, int select_bit, bool scaled,
                     std::vector<double>* grad_scale, const PauliFrame* frame, std::vector<int8_t>* grad_sign) {
  if (select_bit < 0) select_bit = n;
  auto bit = [&](int q) { return q + (q >= select_bit ? 1 : 0); };   // index bit of qubit q in the joint array
  double sigma = 1.0;   // stored amplitudes = true amplitudes / sigma
  size_t rot = frame ? frame->rot.size() : 0;
  int since = 0;        // scaled steps since the last scalar; in a frame each divides by 1/sqrt 2 or more
  constexpr int kScalarEvery = 120;
  for (size_t i = ops.size(); i-- > 0;) {
    const AnsatzOp& o = ops[i];
    int gen[3], par[3];
    const int nr = rotations_of(o, gen, par);
    if (nr) {
      for (int r = nr - 1; r >= 0; --r) {   // last rotation of the gate first
        const double th = params[par[r]];
        const PauliFrame::Rot* fr = frame ? &frame->rot[--rot] : nullptr;
        cdd md[4];
        uint8_t form = GRAD_PLAIN;
        double kappa = 1.0;
        if (gen[r] == 2) {
          // exp(+i th Z / 2) divided by its row-0 phase: diag(1, e^{-i th})
          form = GRAD_PHASE;
          md[0] = 1.0; md[1] = 0.0; md[2] = 0.0; md[3] = cdd(std::cos(th), fr ? -fr->sign * std::sin(th) : -std::sin(th));
        } else if (scaled) {
          const double c = fr ? fr->c : std::cos(th / 2.0), s = fr ? fr->s : std::sin(th / 2.0);
          const cdd j = gen[r] == 0 ? cdd(0.0, 1.0) : cdd(1.0, 0.0);   // X: i s off the diagonal; Y: +s, -s
          const cdd jl = gen[r] == 0 ? cdd(0.0, 1.0) : cdd(-1.0, 0.0);
          if (std::fabs(c) >= std::fabs(s)) {
            form = GRAD_TAN;
            kappa = c;
            const double t = s / c;
            md[0] = 1.0; md[1] = j * t; md[2] = jl * t; md[3] = 1.0;
          } else {
            form = GRAD_COT;
            kappa = s;
            const double u = c / s;
            md[0] = u; md[1] = j; md[2] = jl; md[3] = u;
          }
        } else {
          cdd m[4];
          rotation(gen[r], th, m);
          dagger2(m, md);
        }
        SchedOp g{};
        g.k = 2;
        g.q[0] = (uint8_t)select_bit;     // psi / lambda select bit
        g.q[1] = (uint8_t)bit(o.q0);
        g.grad = 1;
        g.gen = (uint8_t)gen[r];
        g.rot = form;
        g.gidx = (uint32_t)grad_param.size();
        g.dense = g.mat = (uint32_t)pool.size();
        for (int j = 0; j < 4; ++j) pool.push_back({md[j].real(), md[j].imag()});
        g.smul = kappa;
        out.push_back(g);
        grad_param.push_back(par[r]);
        if (grad_scale) grad_scale->push_back(sigma * sigma);
        if (grad_sign) grad_sign->push_back(fr ? (int8_t)fr->sign : (int8_t)1);
        sigma *= kappa;
        if (scaled && gen[r] != 2) ++since;
        if (frame ? since >= kScalarEvery : (std::fabs(sigma) < 0x1p-64 || std::fabs(sigma) > 0x1p64)) {
          since = 0;
          // back to the true scale: every amplitude of both halves times sigma
          const cdd sc[4] = {sigma, 0.0, 0.0, sigma};
          const int q[1] = {bit(o.q0)};
          push_op(out, pool, 1, q, sc);
          out.back().smul = 1.0 / sigma;
          sigma = 1.0;
        }
      }
      continue;
    }
    int k, q[2];
    cdd m[16], md[16];
    fixed_matrix(o, k, q, m);
    const int d = 1 << k;
    for (int r = 0; r < d; ++r)
      for (int c = 0; c < d; ++c) md[r * d + c] = std::conj(m[c * d + r]);
    int qj[2] = {bit(q[0]), k > 1 ? bit(q[1]) : 0};
    push_op(out, pool, k, qj, md);
  }
}

namespace {

// Whether the angles decide which of |c| and |s| is larger in a product of
// neighbouring one-qubit gates of a framed circuit (its rotations have |c| >=
// |s|).  They do not in a run of one X or Y rotation, H or SX (an H or SX with Z
// rotations on one side only: on both, rounding decides between equal moduli),
// nor in RX and RY side by side ((1 + cos a cos b) / 2 >= 1/2).
bool runs_tilt(const std::vector<AnsatzOp>& ops) {
  struct Run { int tilts = 0, gen = -1; bool z = false, z_after = false; };   // gen: 0 X, 1 Y rotation, 2 H or SX
  std::vector<Run> runs(64);
  for (const AnsatzOp& o : ops) {
    if (o.q1 >= 0) {   // a two-qubit gate ends its qubits' runs
      runs[o.q0] = runs[o.q1] = Run{};
      continue;
    }
    Run& r = runs[o.q0];
    auto turn = [&](int gen) {
      if (gen == 3) {   // about Z
        if (r.gen == 2 && r.z) return true;
        (r.tilts ? r.z_after : r.z) = true;
        return false;
      }
      const bool side = r.tilts == 1 && !r.z_after && gen < 2 && r.gen < 2 && gen != r.gen;
      ++r.tilts;
      if (r.tilts > 1 && !side) return true;
      r.gen = gen;
      return false;
    };
    switch (o.kind) {
      case GATE_RX: if (turn(0)) return true; break;
      case GATE_RY: if (turn(1)) return true; break;
      case GATE_RZ: case GATE_P: if (turn(3)) return true; break;
      case GATE_U3: if (turn(3) || turn(1) || turn(3)) return true; break;
      case GATE_H: case GATE_SX: if (turn(2)) return true; break;
      default: break;   // X
    }
  }
  return false;
}

}  // namespace

void adjoint_ops(int n, const std::vector<AnsatzOp>& ops, const double* params, bool backward, bool fuse,
                 bool single_set, AdjointOps& j, bool framed) {
  j.fw.clear(); j.bw.clear(); j.fpool.clear(); j.bpool.clear(); j.grad_param.clear(); j.grad_scale.clear();
  j.grad_sign.clear();
  framed = framed && single_set;
  if (framed) pauli_frame(ops, params, j.frame);
  const PauliFrame* const frame = framed ? &j.frame : nullptr;
  std::vector<SchedOp> raw;
  // a global phase of psi changes neither the energy nor any Im<lambda|P|psi>
  ansatz_forward(n, ops, params, raw, j.fpool, /*phase_free=*/!single_set, frame);
  if (single_set) {
    j.fw = fuse_two_qubit_blocks(raw, j.fpool, true);
    decompose_one_qubit_ops(j.fw, j.fpool, !framed ? DECOMP_BY_ANGLE : runs_tilt(ops) ? DECOMP_STEADY_ENDS : DECOMP_STEADY_SCALARS);
    normalize_one_qubit_ops(j.fw, j.fpool);
  } else {
    // forms that do not depend on the angles, every gate alone: RY (and any
    // real gate) a real 2x2 (4 FMAs per amplitude), RZ diag(1, e^{i th}) (2),
    // CZ / CX renamings -- cheaper than fused 4x4 blocks (16); `fuse` = false
    // keeps the plain matrices
    j.fw = raw;
    if (!fuse) {
      raw.clear();
      j.fpool.clear();
      ansatz_forward(n, ops, params, raw, j.fpool, false);
      for (SchedOp& o : raw) o.realm = 0;
      j.fw = raw;
    }
  }
  if (!backward) return;
  raw.clear();
  ansatz_backward(n, ops, params, raw, j.bpool, j.grad_param, n, single_set, &j.grad_scale, frame, &j.grad_sign);   // [psi | lambda]
  j.bw = fuse ? fuse_two_qubit_blocks(raw, j.bpool, single_set) : raw;
}

void exec_grad_scales(const std::vector<PassPlan>* plans, const std::vector<SchedOp>& ops, std::vector<double>& scale) {
  uint32_t nterms = 0;
  for (const SchedOp& o : ops)
    if (o.grad) nterms = std::max(nterms, o.gidx + 1);
  scale.assign(nterms, 1.0);
  double sigma = 1.0;
  auto visit = [&](const SchedOp& o) {
    if (o.grad) scale[o.gidx] = sigma * sigma;
    if (o.smul != 0.0) sigma *= o.smul;
  };
  if (!plans) {
    for (const SchedOp& o : ops) visit(o);
    return;
  }
  for (const PassPlan& pl : *plans)
    for (uint32_t i : pl.src) visit(ops[i]);
}

namespace {

constexpr uint8_t kPermIdentity2 = 0xE4;   // two-qubit monomial whose rows read their own column

// complex elements of an operation in its pass's matrix block
uint32_t pack_elems(const OpDesc& o, int R) {
  switch (o.kind) {
    case OP_GDZ: return 0;
    case OP_DGR: return 1u << R;
    case OP_GRAD2: return 4;
    case OP_M1R: case OP_M1L: case OP_M2R: return 1u << o.k;
    default: return 1u << (2 * o.k);
  }
}

// one operation of a stage on its way through merge_stage_diagonals
struct StageItem {
  OpDesc od;
  uint32_t src;
  uint32_t mask;         // register slots (bits 0..4) and lane bits (8..10) it acts on
  bool diag = false;     // a diagonal: commutes with the other diagonals
  bool term = false;     // a Z adjoint step: its term is taken where its phase acts
  bool primary = true;   // carries the source index (the phases split off a permutation do not)
  DiagFactor f{};
};

uint32_t slot_mask(const OpDesc& o) {
  switch (o.kind) {
    case OP_D1R: case OP_N1R: case OP_R1R: case OP_M1R: return 1u << o.a;
    case OP_D1L: case OP_R1L: case OP_M1L: return 1u << (8 + o.a);
    case OP_D2R: case OP_M2R: case OP_X2R: return (1u << o.a) | (1u << o.b);
    case OP_GRAD2: return 1u << o.b;   // steps on different qubits commute, whatever their select bit
    default: return 0xFFu;
  }
}

// entries of a merged diagonal that are exactly 1 (bits 0..15) and -1 (16..31)
uint32_t diag_units(const std::vector<DiagFactor>& fs, int NV) {
  uint32_t out = 0;
  for (int v = 0; v < NV; ++v) {
    bool unit = true, neg = false;
    for (const DiagFactor& f : fs) {
      const int r = ((v >> f.a) & 1) | (f.k == 2 ? ((v >> f.b) & 1) << 1 : 0);
      if ((f.negs >> r) & 1) neg = !neg;
      else if (!((f.ones >> r) & 1)) unit = false;
    }
    if (unit) out |= neg ? 1u << (16 + v) : 1u << v;
  }
  return out;
}

// the items of one stage: permutations and their phases apart
void stage_items(const PassPlan& pl, const StageDesc& sd, const std::vector<SchedOp>& ops, std::vector<StageItem>& out) {
  for (int i = sd.op0; i < sd.op1; ++i) {
    StageItem it;
    it.od = pl.desc.ops[i];
    it.src = pl.src[i];
    const OpDesc& o = it.od;
    it.mask = slot_mask(o);
    const bool unit = o.flags & OPF_UNIT_PHASE;
    if (o.kind == OP_M1R && !(o.perm & 1)) {
      it.diag = true;
      it.f.a = o.a;
      it.f.k = 1;
      it.f.ones = unit ? 3 : (o.urows & 3);
      it.f.mat[0] = o.mat;
      it.f.mat[1] = o.mat + 1;
    } else if (o.kind == OP_M2R && (o.perm == kPermIdentity2 || !unit)) {
      StageItem ph = it;
      ph.diag = true;
      ph.f.a = o.a;
      ph.f.b = o.b;
      ph.f.k = 2;
      ph.f.negs = unit ? 0 : ops[it.src].nrows;
      ph.f.ones = unit ? 15 : (uint8_t)(o.urows & 15 & ~ph.f.negs);
      for (int r = 0; r < 4; ++r) ph.f.mat[r] = o.mat + r;
      if (o.perm == kPermIdentity2) {
        out.push_back(ph);
        continue;
      }
      it.od.flags |= OPF_UNIT_PHASE;   // the permutation alone, then its phases by output row
      it.od.urows = 15;
      out.push_back(it);
      ph.primary = false;
      out.push_back(ph);
      continue;
    } else if (o.kind == OP_GRAD2 && o.perm == 2 && o.a == 0) {
      it.diag = it.term = true;
      it.f.a = o.b;
      it.f.k = 1;
      it.f.ones = o.flags == GRAD_PHASE ? 1 : 0;
      it.f.mat[0] = o.mat;
      it.f.mat[1] = o.mat + 3;
    }
    out.push_back(it);
  }
}

}  // namespace

// What it saves: FP64 work.  A phase costs 2 multiply-adds per amplitude, the
// |11> phase of a carried CX 1, a CZ 1, a Z step 4; merged over a stage's four
// slots they cost at most 4 x 15/16 together, CZ signs nothing, and the Z terms
// share one product per (psi, lambda) pair.  30-qubit brick-wall of depth 20:
// 2688 -> 1938 multiply-adds per amplitude, 325 -> 306 ms; 28-qubit gradient:
// forward 898 -> 582, backward 1512 -> 1069, 177 -> 172 ms.
void merge_stage_diagonals(std::vector<PassPlan>& plans, const std::vector<SchedOp>& ops) {
  std::vector<StageItem> items;
  std::vector<uint8_t> done;
  std::vector<int> group;
  for (PassPlan& pl : plans) {
    PassDesc& d = pl.desc;
    if (d.R > 4) continue;
    const int NV = 1 << d.R;
    std::vector<OpDesc> nops;
    std::vector<uint32_t> nsrc, nterm;
    std::vector<std::vector<DiagFactor>> diag;
    std::vector<std::pair<uint16_t, uint16_t>> range(d.nstages);
    nops.reserve(d.nops + d.nops / 2);
    nsrc.reserve(d.nops);
    for (int s = 0; s < d.nstages; ++s) {
      items.clear();
      stage_items(pl, d.st[s], ops, items);
      range[s].first = (uint16_t)nops.size();
      auto emit = [&](const OpDesc& o) {
        nops.push_back(o);
        if (o.kind == OP_GRAD2) {   // gradient rows are numbered in the order the operations run
          nops.back().gidx = (uint32_t)nterm.size();
          nterm.push_back(d.grad_term[o.gidx]);
        }
      };
      size_t left = items.size();
      done.assign(items.size(), 0);
      while (left) {
        // everything that is not a diagonal and waits for nothing before it
        bool progress = true;
        while (progress) {
          progress = false;
          uint32_t before = 0;
          for (size_t i = 0; i < items.size(); ++i) {
            if (done[i]) continue;
            if (!items[i].diag && !(items[i].mask & before)) {
              emit(items[i].od);
              nsrc.push_back(items[i].src);
              done[i] = 1;
              --left;
              progress = true;
            } else {
              before |= items[i].mask;
            }
          }
        }
        // then every diagonal with only diagonals before it on its slots
        group.clear();
        uint32_t blocked = 0;
        for (size_t i = 0; i < items.size(); ++i) {
          if (done[i]) continue;
          if (!items[i].diag) blocked |= items[i].mask;
          else if (!(items[i].mask & blocked)) group.push_back((int)i);
        }
        if (group.empty()) break;   // left == 0: the first item left waits for nothing
        for (int i : group) {
          done[i] = 1;
          --left;
        }
        if (group.size() == 1 && items[group[0]].primary && !items[group[0]].f.negs) {
          emit(items[group[0]].od);
          nsrc.push_back(items[group[0]].src);
          continue;
        }
        // gradient terms first (one OP_GDZ takes each slot once), then the phases
        std::vector<int> terms;
        for (int i : group)
          if (items[i].term) terms.push_back(i);
        while (!terms.empty()) {
          int by_slot[kMaxK] = {-1, -1, -1, -1, -1};
          std::vector<int> later;
          for (int i : terms) {
            if (by_slot[items[i].f.a] < 0) by_slot[items[i].f.a] = i;
            else later.push_back(i);
          }
          OpDesc g{};
          g.kind = OP_GDZ;
          g.k = 1;
          g.gidx = (uint32_t)nterm.size();
          for (int sl = 0; sl < kMaxK; ++sl)
            if (by_slot[sl] >= 0) {
              g.flags |= (uint8_t)(1u << sl);
              nterm.push_back(d.grad_term[items[by_slot[sl]].od.gidx]);
              nsrc.push_back(items[by_slot[sl]].src);
            }
          nops.push_back(g);
          terms.swap(later);
        }
        OpDesc m{};
        m.kind = OP_DGR;
        m.k = 1;
        m.mat = (uint32_t)diag.size();
        std::vector<DiagFactor> fs;
        for (int i : group) {
          fs.push_back(items[i].f);
          m.flags |= (uint8_t)((1u << items[i].f.a) | (items[i].f.k == 2 ? 1u << items[i].f.b : 0u));
          if (items[i].primary && !items[i].term) nsrc.push_back(items[i].src);
        }
        m.gidx = diag_units(fs, NV);
        if ((m.gidx & 0xFFFFu) == (1u << NV) - 1u) continue;   // the identity
        nops.push_back(m);
        diag.push_back(std::move(fs));
      }
      range[s].second = (uint16_t)nops.size();
    }
    size_t elems = 0;
    for (const OpDesc& o : nops) elems += pack_elems(o, d.R);
    if (nops.size() > (size_t)kMaxPassOps || elems > (size_t)kSmemMatElems) continue;
    std::copy(nops.begin(), nops.end(), d.ops);
    d.nops = (uint32_t)nops.size();
    for (int s = 0; s < d.nstages; ++s) {
      d.st[s].op0 = range[s].first;
      d.st[s].op1 = range[s].second;
    }
    std::copy(nterm.begin(), nterm.end(), d.grad_term);
    pl.src = std::move(nsrc);
    pl.diag = std::move(diag);
  }
}

double pass_time_model(const PassDesc& d) {
  double f = 0.0;   // real multiply-adds per amplitude
  for (uint32_t i = 0; i < d.nops; ++i) {
    const OpDesc& o = d.ops[i];
    const bool unit = o.flags & OPF_UNIT_PHASE;
    const int rows = 1 << o.k;
    switch (o.kind) {
      case OP_M1R: case OP_M2R:
        if (!unit) f += 4.0 * (rows - __builtin_popcount(o.urows & ((1u << rows) - 1))) / rows;
        break;
      case OP_M1L: f += unit ? 0.0 : 4.0; break;
      case OP_R1R: case OP_R1L: f += 2.0; break;
      case OP_D1R: case OP_D1L: f += (o.flags & OPF_REAL) ? 4.0 : 8.0; break;
      case OP_N1R: f += 6.0; break;
      case OP_X2R: f += ((o.flags & 1) ? 2.0 : 4.0) + ((o.flags & 2) ? 1.0 : 2.0); break;
      case OP_DGR: f += 4.0 * ((1 << d.R) - __builtin_popcount(o.gidx)) / (1 << d.R); break;
      case OP_GDZ: f += 1.4; break;
      case OP_GRAD2: f += (o.perm == 2 || o.flags) ? 4.0 : 6.0; break;
      default: f += 4.0 * rows; break;
    }
  }
  return std::max(5.75, 0.78 * (0.065 * f + 1.02 * (d.nstages + 1)));
}

void pack_recipe(std::vector<PassPlan>& plans, PackRecipe& r) {
  r.base.clear();
  r.mults.clear();
  for (auto& pl : plans) {
    PassDesc& d = pl.desc;
    const uint32_t base = (uint32_t)r.base.size();
    for (uint32_t i = 0; i < d.nops; ++i) {
      OpDesc& od = d.ops[i];
      const uint32_t rel = (uint32_t)r.base.size() - base;
      if (od.kind == OP_DGR) {
        for (int v = 0; v < (1 << d.R); ++v) {
          const uint32_t at = (uint32_t)r.base.size();
          bool first = true, neg = false;
          r.base.push_back(kPackOne);
          for (const DiagFactor& f : pl.diag[od.mat]) {
            const int row = ((v >> f.a) & 1) | (f.k == 2 ? ((v >> f.b) & 1) << 1 : 0);
            if ((f.ones >> row) & 1) continue;
            if ((f.negs >> row) & 1) { neg = !neg; continue; }
            if (first) r.base[at] = f.mat[row];
            else r.mults.push_back({at, f.mat[row]});
            first = false;
          }
          if (neg) {
            if (!first) r.mults.push_back({at, kPackMinusOne});
            else r.base[at] = kPackMinusOne;
          }
        }
      } else {
        const uint32_t n = pack_elems(od, d.R);
        for (uint32_t e = 0; e < n; ++e) r.base.push_back(od.mat + e);
      }
      od.mat = rel;
    }
    d.mat_base = base;
    d.mat_elems = (uint32_t)r.base.size() - base;
  }
}

void PackRecipe::fill(const cplx64* pool, cplx64* dst) const {
  auto at = [&](uint32_t i) {
    return i == kPackOne ? cplx64{1.0, 0.0} : (i == kPackMinusOne ? cplx64{-1.0, 0.0} : pool[i]);
  };
  for (size_t i = 0; i < base.size(); ++i) dst[i] = at(base[i]);
  // an element's factors follow each other; their product is rounded once (an
  // entry's error is shared by every amplitude it multiplies)
  for (size_t k = 0; k < mults.size();) {
    const uint32_t i = mults[k].first;
    WideScalar w{dst[i].re, dst[i].im};
    for (; k < mults.size() && mults[k].first == i; ++k) w.times(at(mults[k].second));
    dst[i] = w.rounded();
  }
}

void pack_pass_matrices(std::vector<PassPlan>& plans, const cplx64* pool, std::vector<cplx64>& packed) {
  PackRecipe r;
  pack_recipe(plans, r);
  packed.resize(r.base.size());
  r.fill(pool, packed.data());
}

}  // namespace iqb
