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

// max_chain: runs linked by pushed rotations, at most kRotChain.
inline RotPlanHost build_rot_plan(int n, const std::vector<Gate>& gates, int max_chain) {
  // A run whose gates are single-axis rotations about at most two axes in turn (`letters`, equal
  // neighbours merged) stays as one operation per axis: 4 instructions each, no more than any
  // other form, and only their own overlaps.  Every other run is a general 2x2 unitary.
  struct Run {
    int qubit;
    std::vector<int> members;
    bool general;
    int push = kAxisNone, next = -1, prev = -1, depth = 0;
  };
  std::vector<Run> runs;
  struct Event {
    int run, axis;  // a run (run >= 0), or a two-qubit gate and its commuting axis on this qubit
  };
  std::vector<std::vector<Event>> events(n);
  std::vector<int> open(n, -1), run_of(gates.size(), -1);
  for (int g = 0; g < (int)gates.size(); g++) {
    const Gate& gt = gates[g];
    if (gate_controlled(gt.type)) {
      events[gt.target].push_back({-1, rot_commuting_axis(gt.type, false)});
      events[gt.control].push_back({-1, rot_commuting_axis(gt.type, true)});
      open[gt.target] = open[gt.control] = -1;
      continue;
    }
    const int q = gt.target;
    if (open[q] < 0) {
      open[q] = (int)runs.size();
      runs.push_back({q, {}, false});
      events[q].push_back({open[q], 0});
    }
    runs[open[q]].members.push_back(g);
    run_of[g] = open[q];
  }
  for (Run& r : runs) {
    int letters = 0, last = kAxisNone;
    for (int g : r.members) {
      if (gates[g].type == G_U3) {
        r.general = true;
      } else if (rot_letter(gates[g].type) != last) {
        last = rot_letter(gates[g].type);
        letters++;
      }
    }
    if (letters > 2) r.general = true;
  }
  // A general run pushes into the next run of its qubit if that run is general too and every
  // two-qubit gate between them commutes with the same axis.  Chains end after max_chain runs:
  // their numbers are made one after another, and the run that ends a chain costs 4 products more
  // per pair and vector.
  for (int q = 0; q < n; q++) {
    const std::vector<Event>& ev = events[q];
    for (size_t i = 0; i < ev.size(); i++) {
      if (ev[i].run < 0 || !runs[ev[i].run].general) continue;
      int axis = kAxisNone;
      size_t j = i + 1;
      for (; j < ev.size() && ev[j].run < 0; j++) {
        if (axis == kAxisNone) axis = ev[j].axis;
        if (ev[j].axis != axis) break;
      }
      if (j >= ev.size() || ev[j].run < 0) continue;
      Run& r = runs[ev[i].run];
      Run& s = runs[ev[j].run];
      if (!s.general || r.depth + 1 >= max_chain) continue;
      r.push = axis;
      r.next = ev[j].run;
      s.prev = ev[i].run;
      s.depth = r.depth + 1;
    }
  }
  RotPlanHost pl;
  struct Item {  // what becomes a RotRun: op index, members, links to other items
    RotRun r;
    int next;
  };
  std::vector<Item> items;
  std::vector<int> item_of(runs.size(), -1);
  auto add_op = [&](int kind, int target, int control, int mask, int anchor) {
    const RotStep st = {kind, target, control, pl.noverlaps, mask, anchor};
    for (int m = mask; m; m &= m - 1) pl.noverlaps++;
    pl.steps.push_back(st);
    return st;
  };
  std::vector<std::vector<int>> item_members;
  auto add_item = [&](const RotStep& op, const std::vector<int>& members, int push, bool pulled) {
    items.push_back({{(int)pl.steps.size() - 1, 0, (int)members.size(), push, pulled ? 1 : 0, op.kind, op.coff, op.mask,
                      members.size() == 1 && gates[members[0]].type == G_U3 ? 1 : 0, -1},
                     -1});
    item_members.push_back(members);
    return (int)items.size() - 1;
  };
  for (int g = 0; g < (int)gates.size(); g++) {
    const Gate& gt = gates[g];
    if (gate_controlled(gt.type)) {
      const bool cry = gt.type == G_CRY;
      const RotStep op = add_op(cry ? kOpCry : gt.type == G_CNOT ? kOpCnot : kOpCz, gt.target, gt.control, cry ? 2 : 0, g);
      if (cry) add_item(op, {g}, kAxisNone, false);
      continue;
    }
    const Run& r = runs[run_of[g]];
    if (r.members.back() != g) continue;  // the run takes its last gate's place
    if (r.general) {
      // pushed axis: measured by the run that it is pushed into
      const int mask = r.push == kAxisX ? 6 : r.push == kAxisY ? 5 : r.push == kAxisZ ? 3 : 7;
      const int kind = kOpRot | kOpZi | (r.push == kAxisY ? kOpX : 0) | (r.push == kAxisNone ? kOpZo : 0);
      item_of[run_of[g]] = add_item(add_op(kind, r.qubit, -1, mask, g), r.members, r.push, r.prev >= 0);
      continue;
    }
    for (size_t i = 0; i < r.members.size();) {
      const int axis = rot_letter(gates[r.members[i]].type);
      std::vector<int> same;
      for (; i < r.members.size() && rot_letter(gates[r.members[i]].type) == axis; i++) same.push_back(r.members[i]);
      const int kind = axis == kAxisZ ? kOpPhase : axis == kAxisX ? kOpRot | kOpX : kOpRot;
      add_item(add_op(kind, r.qubit, -1, 1 << (axis - 1), g), same, kAxisNone, false);
    }
  }
  for (size_t i = 0; i < runs.size(); i++)
    if (runs[i].next >= 0) items[item_of[i]].next = item_of[runs[i].next];
  // chain order: every chain contiguous and within one CTA, whose parameters are listed together
  auto gate_params = [&](int j) {
    int np = 0;
    for (int g : item_members[j]) np += gate_param_num(gates[g].type);
    return np;
  };
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
      np += gate_params(j);
    }
    const bool listed = np <= kRotParams;  // else the chain's threads take them one by one
    if ((int)pl.runs.size() + len - pl.cta.back() > kRotThreads ||
        (listed && (int)pl.params.size() + np - pl.cta_params.back() > kRotParams))
      close_cta();
    for (int j = (int)i; j >= 0; j = items[j].next) {
      RotRun r = items[j].r;
      r.first = (int)pl.members.size();
      r.soff = listed ? (int)pl.params.size() - pl.cta_params.back() : -1;
      for (int g : item_members[j]) {
        pl.members.push_back(g);
        for (int k = 0; listed && k < gate_param_num(gates[g].type); k++) pl.params.push_back(gates[g].pstart + k);
      }
      pl.runs.push_back(r);
    }
  }
  if ((int)pl.runs.size() > pl.cta.back()) close_cta();
  for (int longer = 1; longer >= 0; longer--)
    for (int i = 0; i < (int)pl.runs.size(); i++)
      if (!pl.runs[i].pulled && (pl.runs[i].push != kAxisNone) == (longer == 1)) pl.heads.push_back(i);
  return pl;
}

// Steps [k0, k1) as operations on n qubits, qubit q of a step being loc[q]; appended to ops.
// ends receives n places (RotPlan::ends).
inline void lower_rot_steps(const std::vector<RotStep>& steps, int k0, int k1, int n, const std::vector<int>& loc,
                            std::vector<RotOp>& ops, std::vector<int>& ends) {
  // qubit q of the amplitude at place p is the parity of p & row[q]; the amplitude with bit q
  // changed is at p ^ pair[q].  A CNOT adds its control's row to its target's.
  unsigned row[32], pair[32];
  for (int q = 0; q < n; q++) row[q] = pair[q] = 1u << q;
  struct Cz {
    unsigned a, b;
  };
  std::vector<Cz> waiting;
  auto odd = [](unsigned v) { return __builtin_popcount(v) & 1; };
  auto emit_cz = [&](const Cz& z) {
    RotOp op = {};
    op.kind = kOpCz;
    op.cz0 = (unsigned short)z.a;
    op.cz1 = (unsigned short)z.b;
    ops.push_back(op);
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
      waiting.push_back({row[t], row[c]});
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
      for (size_t i = 0; i < waiting.size();) {
        const Cz z = waiting[i];
        if (!odd(z.a & pair[t]) && !odd(z.b & pair[t])) {
          i++;
          continue;
        }
        waiting.erase(waiting.begin() + i);
        if (first && s.kind != kOpCry) {  // a CRY visits half of the places only
          op.cz0 = (unsigned short)z.a;
          op.cz1 = (unsigned short)z.b;
          first = false;
        } else {
          emit_cz(z);
        }
      }
    }
    ops.push_back(op);
  }
  for (const Cz& z : waiting) emit_cz(z);
  for (int q = 0; q < n; q++) ends.push_back((int)pair[q]);
}

}  // namespace sqg
