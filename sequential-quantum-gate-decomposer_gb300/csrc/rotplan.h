// Host side of the rotation plan (rot.cuh): which operations a gate list becomes.  It depends
// on the gate list alone and is made once per circuit handle.
#pragma once
#include <algorithm>
#include <vector>

#include "rot.cuh"

namespace sqg {

// An operation before its qubits become masks; its index is that of its numbers.
struct RotStep {
  int kind, target, control, coff, mask;
  int anchor;  // gate whose place it takes (the last gate of its run)
};

struct RotPlanHost {
  std::vector<RotStep> steps;
  std::vector<RotRun> runs;
  std::vector<int> members, cta, params, cta_params, heads;
  int noverlaps = 0;
};

// Axis that commutes with a two-qubit gate on its target or control qubit.
inline int rot_commuting_axis(int type, bool on_control) {
  if (on_control || type == G_CZ) return kAxisZ;
  return type == G_CNOT ? kAxisX : kAxisY;
}

inline int rot_letter(int type) { return type == G_RX ? kAxisX : type == G_RY ? kAxisY : kAxisZ; }

// The runs of a gate list, in the order of their first gates.  Run r's gates are members[first[r] ..
// first[r + 1]); before: the run in front of it on its qubit (-1: none); between: the axis that commutes
// with every two-qubit gate since then (kAxisNone: there is none such).  general: a 2x2 unitary; else the
// gates are single-axis rotations about at most two axes in turn (equal neighbours merged), which stay as
// one operation per axis: 4 instructions each, no more than any other form, and only their own overlaps.
struct RotRuns {
  struct Run {
    int qubit, first, count, before, between, last;  // last: its last gate
    bool general;
  };
  std::vector<Run> runs;
  std::vector<int> members;
  std::vector<int> run_of;  // of a gate; controlled gates: -1
};

inline RotRuns find_rot_runs(int n, const std::vector<Gate>& gates) {
  RotRuns rr;
  const int L = (int)gates.size();
  rr.run_of.assign(L, -1);
  std::vector<int> open(n, -1), latest(n, -1), axis(n, -1);  // axis: -1 no two-qubit gate since `latest`
  int singles = 0;
  auto meet = [&](int q, int a) {
    open[q] = -1;
    axis[q] = axis[q] < 0 || axis[q] == a ? a : kAxisNone;
  };
  for (int g = 0; g < L; g++) {
    const Gate& gt = gates[g];
    if (gate_controlled(gt.type)) {
      meet(gt.target, rot_commuting_axis(gt.type, false));
      meet(gt.control, rot_commuting_axis(gt.type, true));
      continue;
    }
    const int q = gt.target;
    if (open[q] < 0) {
      open[q] = (int)rr.runs.size();
      rr.runs.push_back({q, 0, 0, latest[q], std::max(axis[q], 0), g, false});
      latest[q] = open[q];
      axis[q] = -1;
    }
    rr.runs[open[q]].count++;
    rr.runs[open[q]].last = g;
    rr.run_of[g] = open[q];
    singles++;
  }
  int at = 0;
  for (RotRuns::Run& r : rr.runs) {
    r.first = at;
    at += r.count;
    r.count = 0;
  }
  rr.members.resize(singles);
  for (int g = 0; g < L; g++)
    if (rr.run_of[g] >= 0) {
      RotRuns::Run& r = rr.runs[rr.run_of[g]];
      rr.members[r.first + r.count++] = g;
    }
  for (RotRuns::Run& r : rr.runs) {
    int letters = 0, last = kAxisNone;
    for (int m = r.first; m < r.first + r.count; m++) {
      const int type = gates[rr.members[m]].type;
      if (type == G_U3) {
        r.general = true;
      } else if (rot_letter(type) != last) {
        last = rot_letter(type);
        letters++;
      }
    }
    if (letters > 2) r.general = true;
  }
  return rr;
}

// A general run pushes into the next run of its qubit if that run is general too and every
// two-qubit gate between them commutes with the same axis.  Chains end after max_chain (at most
// kRotChain) runs: their numbers are made one after another, and the run that ends a chain costs 4
// products more per pair and vector.
inline RotPlanHost build_rot_plan(const RotRuns& rr, const std::vector<Gate>& gates, int max_chain) {
  const int L = (int)gates.size(), nruns = (int)rr.runs.size();
  struct Link {
    int push = kAxisNone, pulled = kAxisNone, next = -1, depth = 0;
  };
  std::vector<Link> links(nruns);
  for (int r = 0; r < nruns; r++) {
    const RotRuns::Run& run = rr.runs[r];
    if (!run.general || run.before < 0 || run.between == kAxisNone || !rr.runs[run.before].general) continue;
    Link& b = links[run.before];
    if (b.depth + 1 >= max_chain) continue;
    b.push = run.between;
    b.next = r;
    links[r].pulled = run.between;
    links[r].depth = b.depth + 1;
  }
  RotPlanHost pl;
  pl.steps.reserve(L);
  struct Item {  // what becomes a RotRun: its gates, a range of rr.members or the one gate `lone`; the next of its chain
    RotRun r;
    int lone, nparams, next;
  };
  std::vector<Item> items;
  items.reserve(L);
  std::vector<int> item_of(nruns, -1);
  auto add_op = [&](int kind, int target, int control, int mask, int anchor) {
    pl.steps.push_back({kind, target, control, pl.noverlaps, mask, anchor});
    pl.noverlaps += (mask & 1) + (mask >> 1 & 1) + (mask >> 2);
  };
  auto add_item = [&](int first, int count, int lone, int push, int pulled) {  // pulled: its axis
    const RotStep& op = pl.steps.back();
    auto member = [&](int k) { return lone >= 0 ? lone : rr.members[first + k]; };
    int np = 0;
    for (int k = 0; k < count; k++) np += gate_param_num(gates[member(k)].type);
    const bool z = (push == kAxisNone || push == kAxisZ) && (pulled == kAxisNone || pulled == kAxisZ);
    const int lone_u3 = z && count == 1 && gates[member(0)].type == G_U3 ? 1 : 0;
    items.push_back({{(int)pl.steps.size() - 1, first, count, push, pulled != kAxisNone ? 1 : 0, op.kind, op.coff, op.mask, lone_u3, -1},
                     lone, np, -1});
    return (int)items.size() - 1;
  };
  for (int g = 0; g < L; g++) {
    const Gate& gt = gates[g];
    if (gate_controlled(gt.type)) {
      const bool cry = gt.type == G_CRY;
      add_op(cry ? kOpCry : gt.type == G_CNOT ? kOpCnot : kOpCz, gt.target, gt.control, cry ? 2 : 0, g);
      if (cry) add_item(0, 1, g, kAxisNone, kAxisNone);
      continue;
    }
    const RotRuns::Run& r = rr.runs[rr.run_of[g]];
    if (r.last != g) continue;  // the run takes its last gate's place
    const Link& l = links[rr.run_of[g]];
    if (r.general) {
      // pushed axis: measured by the run that it is pushed into
      const int mask = l.push == kAxisX ? 6 : l.push == kAxisY ? 5 : l.push == kAxisZ ? 3 : 7;
      add_op(kOpRot | kOpZi | (l.push == kAxisY ? kOpX : 0) | (l.push == kAxisNone ? kOpZo : 0), r.qubit, -1, mask, g);
      item_of[rr.run_of[g]] = add_item(r.first, r.count, -1, l.push, l.pulled);
      continue;
    }
    for (int m = r.first, end = r.first + r.count; m < end;) {
      const int axis = rot_letter(gates[rr.members[m]].type), m0 = m;
      while (m < end && rot_letter(gates[rr.members[m]].type) == axis) m++;
      const int kind = axis == kAxisZ ? kOpPhase : axis == kAxisX ? kOpRot | kOpX : kOpRot;
      add_op(kind, r.qubit, -1, 1 << (axis - 1), g);
      add_item(m0, m - m0, -1, kAxisNone, kAxisNone);
    }
  }
  for (int r = 0; r < nruns; r++)
    if (links[r].next >= 0) items[item_of[r]].next = item_of[links[r].next];
  // chain order: every chain contiguous and within one CTA, whose parameters are listed together
  pl.runs.reserve(items.size());
  pl.members.reserve(L);
  pl.params.reserve(3 * (size_t)L);
  pl.cta.push_back(0);
  pl.cta_params.push_back(0);
  auto close_cta = [&]() {
    pl.cta.push_back((int)pl.runs.size());
    pl.cta_params.push_back((int)pl.params.size());
  };
  for (size_t i = 0; i < items.size(); i++) {
    if (items[i].r.pulled) continue;
    int len = 0, np = 0;
    for (int j = (int)i; j >= 0; j = items[j].next) {
      len++;
      np += items[j].nparams;
    }
    const bool listed = np <= kRotParams;  // else the chain's threads take them one by one
    if ((int)pl.runs.size() + len - pl.cta.back() > kRotThreads ||
        (listed && (int)pl.params.size() + np - pl.cta_params.back() > kRotParams))
      close_cta();
    for (int j = (int)i; j >= 0; j = items[j].next) {
      RotRun r = items[j].r;
      r.soff = listed ? (int)pl.params.size() - pl.cta_params.back() : -1;
      const int first = r.first;
      r.first = (int)pl.members.size();
      for (int m = 0; m < r.count; m++) {
        const int g = items[j].lone >= 0 ? items[j].lone : rr.members[first + m];
        pl.members.push_back(g);
        for (int k = 0; listed && k < gate_param_num(gates[g].type); k++) pl.params.push_back(gates[g].pstart + k);
      }
      pl.runs.push_back(r);
    }
  }
  if ((int)pl.runs.size() > pl.cta.back()) close_cta();
  pl.heads.reserve(pl.runs.size());
  for (int longer = 1; longer >= 0; longer--)
    for (int i = 0; i < (int)pl.runs.size(); i++)
      if (!pl.runs[i].pulled && (pl.runs[i].push != kAxisNone) == (longer == 1)) pl.heads.push_back(i);
  return pl;
}

// A CZ by the rows of its two qubits.
struct RotCz {
  unsigned a, b;
};

// Steps [k0, k1) as operations on n qubits, qubit q of a step being loc[q]; appended to ops.
// ends receives n places (RotPlan::ends); waiting is scratch.
inline void lower_rot_steps(const std::vector<RotStep>& steps, int k0, int k1, int n, const std::vector<int>& loc,
                            std::vector<RotOp>& ops, std::vector<int>& ends, std::vector<RotCz>& waiting) {
  // qubit q of the amplitude at place p is the parity of p & row[q]; the amplitude with bit q
  // changed is at p ^ pair[q].  A CNOT adds its control's row to its target's.
  unsigned row[32], pair[32];
  for (int q = 0; q < n; q++) row[q] = pair[q] = 1u << q;
  // CZs that no operation has met yet; one that comes twice is none.  At most kWaiting of them (all pairs of
  // 13 qubits are 78), so that a long circuit is not walked for each: the oldest goes its own way then.
  constexpr size_t kWaiting = 96;
  waiting.clear();
  auto odd = [](unsigned v) { return __builtin_parity(v); };
  auto emit_cz = [&](const RotCz& z) {
    RotOp op = {};
    op.kind = kOpCz;
    op.cz0 = (unsigned short)z.a;
    op.cz1 = (unsigned short)z.b;
    ops.push_back(op);
  };
  auto add_cz = [&](const RotCz& z) {
    for (RotCz& w : waiting)
      if ((w.a == z.a && w.b == z.b) || (w.a == z.b && w.b == z.a)) {
        waiting.erase(waiting.begin() + (&w - waiting.data()));
        return;
      }
    if (waiting.size() == kWaiting) {
      emit_cz(waiting[0]);
      waiting.erase(waiting.begin());
    }
    waiting.push_back(z);
  };
  for (int k = k0; k < k1; k++) {
    const RotStep& s = steps[k];
    const int t = loc[s.target], c = s.control >= 0 ? loc[s.control] : -1;
    if (s.kind == kOpCnot) {
      row[t] ^= row[c];
      pair[c] ^= pair[t];
      continue;
    }
    if (s.kind == kOpCz) {
      add_cz({row[t], row[c]});
      continue;
    }
    RotOp op = {};
    op.kind = s.kind;
    op.rec = k;
    op.coff = s.coff;
    op.mask = s.mask;
    op.pair = (unsigned short)pair[t];
    op.row = (unsigned short)row[t];
    // the highest bit of the pair mask numbers the pairs: the lower ones then run through
    // consecutive places, without bank conflicts
    op.b0 = (unsigned short)(31 - __builtin_clz(pair[t]));
    if (s.kind == kOpCry) {
      op.crow = (unsigned short)row[c];
      op.b1 = (unsigned short)(31 - __builtin_clz(row[c] & ~(1u << op.b0)));
    }
    if (s.kind != kOpPhase) {  // diagonal operations commute with every CZ
      bool first = true;
      size_t kept = 0;
      for (const RotCz& z : waiting) {
        if (!odd(z.a & pair[t]) && !odd(z.b & pair[t])) {
          waiting[kept++] = z;
        } else if (first && s.kind != kOpCry) {  // a CRY visits half of the places only
          op.cz0 = (unsigned short)z.a;
          op.cz1 = (unsigned short)z.b;
          first = false;
        } else {
          emit_cz(z);
        }
      }
      waiting.resize(kept);
    }
    ops.push_back(op);
  }
  for (const RotCz& z : waiting) emit_cz(z);
  for (int q = 0; q < n; q++) ends.push_back((int)pair[q]);
}

}  // namespace sqg
