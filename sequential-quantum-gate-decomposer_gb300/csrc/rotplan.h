// Host side of the rotation plan (rot.cuh): which operations a gate list becomes.  It depends
// on the gate list alone and is made once per circuit handle.
#pragma once
#include <algorithm>
#include <vector>

#include "rot.cuh"

namespace sqg {

struct RotPlanHost {
  std::vector<RotOp> ops;
  std::vector<int> anchor;  // gate whose place an operation takes (the last gate of its run)
  std::vector<RotRun> runs;
  std::vector<int> members, cta;
  int noverlaps = 0;
};

// Axis that commutes with a two-qubit gate on its target or control qubit.
inline int rot_commuting_axis(int type, bool on_control) {
  if (on_control || type == G_CZ) return kAxisZ;
  return type == G_CNOT ? kAxisX : kAxisY;
}

inline int rot_letter(int type) { return type == G_RX ? kAxisX : type == G_RY ? kAxisY : kAxisZ; }

inline RotPlanHost build_rot_plan(int n, const std::vector<Gate>& gates) {
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
  // two-qubit gate between them commutes with the same axis.  Chains end after kRotChain runs:
  // their numbers are made one after another, and the run that ends a chain costs 4
  // instructions more per pair (3 % at 16).
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
      if (!s.general || r.depth + 1 >= kRotChain) continue;
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
    RotOp op = {kind, target | (std::max(control, 0) << 8), pl.noverlaps, mask};
    for (int m = mask; m; m &= m - 1) pl.noverlaps++;
    pl.ops.push_back(op);
    pl.anchor.push_back(anchor);
    return op;
  };
  std::vector<std::vector<int>> item_members;
  auto add_item = [&](const RotOp& op, const std::vector<int>& members, int push, bool pulled) {
    items.push_back({{(int)pl.ops.size() - 1, 0, (int)members.size(), push, pulled ? 1 : 0, op.kind, op.coff, op.mask,
                      members.size() == 1 && gates[members[0]].type == G_U3 ? 1 : 0},
                     -1});
    item_members.push_back(members);
    return (int)items.size() - 1;
  };
  for (int g = 0; g < (int)gates.size(); g++) {
    const Gate& gt = gates[g];
    if (gate_controlled(gt.type)) {
      const bool cry = gt.type == G_CRY;
      const RotOp op = add_op(cry ? kOpCry : gt.type == G_CNOT ? kOpCnot : kOpCz, gt.target, gt.control, cry ? 2 : 0, g);
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
  // chain order: every chain contiguous and within one CTA
  pl.cta.push_back(0);
  for (size_t i = 0; i < items.size(); i++) {
    if (items[i].r.pulled) continue;
    int len = 0;
    for (int j = (int)i; j >= 0; j = items[j].next) len++;
    if ((int)pl.runs.size() + len - pl.cta.back() > kRotThreads) pl.cta.push_back((int)pl.runs.size());
    for (int j = (int)i; j >= 0; j = items[j].next) {
      RotRun r = items[j].r;
      r.first = (int)pl.members.size();
      pl.members.insert(pl.members.end(), item_members[j].begin(), item_members[j].end());
      pl.runs.push_back(r);
    }
  }
  if ((int)pl.runs.size() > pl.cta.back()) pl.cta.push_back((int)pl.runs.size());
  return pl;
}

}  // namespace sqg
