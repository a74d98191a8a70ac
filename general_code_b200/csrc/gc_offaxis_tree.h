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

// Nodes in one array, children as linked lists: a vector per node made the tree
// of r <= 4 (252 lines) 82 us of a call, this 12 us; r <= 6 370 and 55 us.
struct LineTree {
  struct Node {
    int step, line, weight; // weight: nodes of the subtree
    int first, next;        // first child, next sibling (-1: none)
  };
  std::vector<Node> t;

  LineTree() { clear(); }
  void clear() { t.assign(1, Node{0, -1, 0, -1, -1}); }

  // The node a line ends on (new nodes are put before their siblings).
  int add(const std::vector<int> &steps) {
    int n = 0;
    for (int e : steps) {
      int c = t[n].first;
      while (c >= 0 && t[c].step != e)
        c = t[c].next;
      if (c < 0) {
        c = (int)t.size();
        t.push_back(Node{e, -1, 0, -1, t[n].first});
        t[n].first = c;
      }
      n = c;
    }
    return n;
  }

  // Children in walking order: the largest subtree last (its products need no
  // stack level below it), the others by size, equal sizes by step. (A node has
  // at most six children, one per step.)
  void order() {
    // children have larger indices than their parent
    for (int n = (int)t.size() - 1; n >= 0; n--) {
      t[n].weight = 1;
      int c[6], k = 0;
      for (int i = t[n].first; i >= 0; i = t[i].next) {
        t[n].weight += t[i].weight;
        int j = k++;
        for (; j > 0 && before(i, c[j - 1]); j--)
          c[j] = c[j - 1];
        c[j] = i;
      }
      for (int j = 0; j < k; j++)
        t[c[j]].next = j + 1 < k ? c[j + 1] : -1;
      t[n].first = k ? c[0] : -1;
    }
  }

private:
  bool before(int a, int b) const {
    return t[a].weight != t[b].weight ? t[a].weight < t[b].weight : t[a].step < t[b].step;
  }
};

// Distinct lines are numbered in tree order; each chunk of at most
// lines_per_chunk of them walks its own part of the tree. L: the spatial
// extents. Nodes are empty when a chunk needs more than stack_levels levels (its
// lines and chunk_lines are there all the same: the caller's other form takes
// its launch ranges from them), or without a walk (stack_levels < 0).
inline OffaxisTree offaxis_tree(const int L[3], const std::vector<OffaxisLine> &lines,
                                int lines_per_chunk, int stack_levels = kTreeStack) {
  OffaxisTree out;
  bool fits = stack_levels >= 0;
  // all distinct lines, numbered in the order of a walk of their tree
  LineTree all;
  std::vector<int> end(lines.size());
  for (size_t i = 0; i < lines.size(); i++) {
    end[i] = all.add(lines[i].pattern);
    if (all.t[end[i]].line < 0)
      all.t[end[i]].line = (int)i; // (a plan line with this pattern)
  }
  all.order();
  std::vector<int> number(all.t.size(), -1), todo{0};
  while (!todo.empty()) { // a node, its children, then its next sibling
    const int n = todo.back();
    todo.pop_back();
    if (all.t[n].line >= 0) {
      number[n] = (int)out.first.size();
      out.first.push_back(all.t[n].line);
    }
    if (all.t[n].next >= 0)
      todo.push_back(all.t[n].next);
    if (all.t[n].first >= 0)
      todo.push_back(all.t[n].first);
  }
  out.distinct.reserve(lines.size());
  for (size_t i = 0; i < lines.size(); i++)
    out.distinct.push_back(number[end[i]]);
  // each chunk of consecutive lines as a walk of its own tree
  const int total = (int)out.first.size();
  LineTree chunk;
  struct Visit {
    int node, parent_level; // stack level of the parent's product, -1: in registers
    int level;              // first free stack level
    int pos[3];             // displacement of the parent's end
  };
  std::vector<Visit> visits;
  for (int l0 = 0; l0 < total; l0 += lines_per_chunk) {
    out.chunk_lines.push_back(l0);
    if (!fits)
      continue;
    const int l1 = std::min(total, l0 + lines_per_chunk);
    chunk.clear();
    for (int l = l0; l < l1; l++) {
      const int n = chunk.add(lines[out.first[l]].pattern);
      chunk.t[n].line = l;
    }
    chunk.order();
    out.chunk_nodes.push_back((int)out.nodes.size());
    // depth first; a node with several children keeps its product on a level
    // until the last of them, which continues from the stack as well
    visits.clear();
    int c[6], k = 0;
    for (int i = chunk.t[0].first; i >= 0; i = chunk.t[i].next)
      c[k++] = i;
    while (k > 0)
      visits.push_back({c[--k], -2, 0, {0, 0, 0}});
    while (!visits.empty()) {
      const Visit v = visits.back();
      visits.pop_back();
      const LineTree::Node &tn = chunk.t[v.node];
      OffaxisNode q{};
      const int axis = std::abs(tn.step) - 1;
      int at[3] = {v.pos[0], v.pos[1], v.pos[2]}, to[3] = {v.pos[0], v.pos[1], v.pos[2]};
      if (tn.step > 0)
        to[axis] += 1;
      else
        at[axis] -= 1, to[axis] -= 1;
      for (int d = 0; d < 3; d++)
        q.d[d] = ((at[d] % L[d]) + L[d]) % L[d];
      q.line = tn.line;
      q.axis = (signed char)axis;
      q.back = tn.step < 0;
      q.from = (signed char)v.parent_level;
      k = 0;
      for (int i = tn.first; i >= 0; i = chunk.t[i].next)
        c[k++] = i;
      q.push = -1;
      if (k > 1) {
        if (v.level >= stack_levels) {
          fits = false;
          break;
        }
        q.push = (signed char)v.level;
      }
      out.nodes.push_back(q);
      for (int i = k; i-- > 0;) {
        // the first child follows at once (registers); the others find the
        // product on the stack, and the last one frees its level
        Visit w{c[i], i == 0 ? -1 : (int)q.push, 0, {to[0], to[1], to[2]}};
        w.level = k > 1 && i + 1 < k ? v.level + 1 : v.level;
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
