// The tree of off-axis lines that gc_offaxis_gauge.cu walks (host code; no CUDA).
//
// Lines with equal step patterns are one line, and lines that begin alike share
// the product of the common steps: the patterns form a tree, one node per step.
#pragma once

#include <algorithm>
#include <cstdlib>
#include <vector>

namespace gc {

// A space line's links, in order (OffaxisLine::pattern, OffaxisLineDesc::s):
// +a steps forward along axis a-1 (1..3), -a steps back and takes the
// link's adjoint.
struct OffaxisLine {
  std::vector<int> pattern;
  int disp[3];
};

// Products that a walk keeps for later branches, at most (a thread's private
// stack in the kernel).
constexpr int kTreeStack = 12;

struct OffaxisNode {
  int d[3];          // site of the node's link, as a residue displacement from the start
  int line;          // distinct line that ends here, or -1
  signed char axis;  // the link's axis
  signed char back;  // 1: a step back (the link's adjoint)
  signed char from;  // product extended: -1 the previous node's, >= 0 that stack level's,
                     // -2 none (first step)
  signed char push;  // stack level that keeps this node's product, or -1
  int pad[3];
};
struct OffaxisTree {
  std::vector<int> distinct;       // plan line -> distinct line
  std::vector<int> first;          // distinct line -> a plan line
  std::vector<OffaxisNode> nodes;  // chunk after chunk
  std::vector<int> chunk_nodes;    // first node of each chunk, and the end
  std::vector<int> chunk_lines;    // first distinct line of each chunk, and the end
};

struct TreeNode {
  int step = 0, line = -1, weight = 0; // weight: nodes of the subtree
  std::vector<int> children;
};

// Children in walking order: the largest subtree last (its products need no
// stack level below it), the others by size, equal sizes by step.
inline void order_children(std::vector<TreeNode> &t, int n) {
  t[n].weight = 1;
  for (int c : t[n].children) {
    order_children(t, c);
    t[n].weight += t[c].weight;
  }
  std::sort(t[n].children.begin(), t[n].children.end(), [&](int a, int b) {
    return t[a].weight != t[b].weight ? t[a].weight < t[b].weight : t[a].step < t[b].step;
  });
}

inline int add_line(std::vector<TreeNode> &t, const std::vector<int> &steps) {
  int n = 0;
  for (int e : steps) {
    int next = -1;
    for (int c : t[n].children)
      if (t[c].step == e)
        next = c;
    if (next < 0) {
      next = (int)t.size();
      t[n].children.push_back(next);
      t.emplace_back();
      t[next].step = e;
    }
    n = next;
  }
  return n;
}

// Distinct lines are numbered in tree order; each chunk of at most
// lines_per_chunk of them walks its own part of the tree. L: the spatial
// extents. Nodes are empty when a chunk needs more than stack_levels levels (its
// lines and chunk_lines are there all the same: the caller's other form takes
// its launch ranges from them).
inline OffaxisTree offaxis_tree(const int L[3], const std::vector<OffaxisLine> &lines,
                                int lines_per_chunk, int stack_levels = kTreeStack) {
  OffaxisTree out;
  bool fits = true;
  // all distinct lines, numbered in the order of a walk of their tree
  std::vector<TreeNode> all(1);
  std::vector<int> end(lines.size());
  for (size_t i = 0; i < lines.size(); i++) {
    end[i] = add_line(all, lines[i].pattern);
    if (all[end[i]].line < 0)
      all[end[i]].line = (int)i; // (a plan line with this pattern)
  }
  order_children(all, 0);
  std::vector<int> number(all.size(), -1), todo{0};
  while (!todo.empty()) {
    const int n = todo.back();
    todo.pop_back();
    if (all[n].line >= 0) {
      number[n] = (int)out.first.size();
      out.first.push_back(all[n].line);
    }
    for (size_t k = all[n].children.size(); k-- > 0;)
      todo.push_back(all[n].children[k]);
  }
  for (size_t i = 0; i < lines.size(); i++)
    out.distinct.push_back(number[end[i]]);
  // each chunk of consecutive lines as a walk of its own tree
  const int total = (int)out.first.size();
  for (int l0 = 0; l0 < total; l0 += lines_per_chunk) {
    const int l1 = std::min(total, l0 + lines_per_chunk);
    std::vector<TreeNode> t(1);
    for (int l = l0; l < l1; l++)
      t[add_line(t, lines[out.first[l]].pattern)].line = l;
    order_children(t, 0);
    out.chunk_nodes.push_back((int)out.nodes.size());
    out.chunk_lines.push_back(l0);
    struct Visit {
      int node, parent_level; // stack level of the parent's product, -1: in registers
      int level;              // first free stack level
      int pos[3];             // displacement of the parent's end
    };
    // depth first; a node with several children keeps its product on a level
    // until the last of them, which continues from the stack as well
    std::vector<Visit> visits;
    for (size_t k = t[0].children.size(); k-- > 0;)
      visits.push_back({t[0].children[k], -2, 0, {0, 0, 0}});
    while (!visits.empty()) {
      const Visit v = visits.back();
      visits.pop_back();
      const TreeNode &tn = t[v.node];
      OffaxisNode q{};
      const int axis = std::abs(tn.step) - 1;
      int at[3] = {v.pos[0], v.pos[1], v.pos[2]}, to[3] = {v.pos[0], v.pos[1], v.pos[2]};
      if (tn.step > 0)
        to[axis] += 1;
      else
        at[axis] -= 1, to[axis] -= 1;
      for (int k = 0; k < 3; k++)
        q.d[k] = ((at[k] % L[k]) + L[k]) % L[k];
      q.line = tn.line;
      q.axis = (signed char)axis;
      q.back = tn.step < 0;
      q.from = (signed char)v.parent_level;
      const size_t nch = tn.children.size();
      q.push = -1;
      if (nch > 1) {
        if (v.level >= stack_levels) {
          fits = false;
          break;
        }
        q.push = (signed char)v.level;
      }
      out.nodes.push_back(q);
      for (size_t k = nch; k-- > 0;) {
        // the first child follows at once (registers); the others find the
        // product on the stack, and the last one frees its level
        Visit w{tn.children[k], k == 0 ? -1 : (int)q.push, 0, {to[0], to[1], to[2]}};
        w.level = nch > 1 && k + 1 < nch ? v.level + 1 : v.level;
        visits.push_back(w);
      }
    }
  }
  out.chunk_nodes.push_back((int)out.nodes.size());
  out.chunk_lines.push_back(total);
  if (!fits) {
    out.nodes.clear();
    out.chunk_nodes.clear();
  }
  return out;
}

} // namespace gc
