"""The tree of off-axis lines (host code): a walk with the kernel's stack rules
gives every line's steps, and a tree that needs more stack levels than there
are still lists every line and chunk, since the exact form takes its launches
from them.
"""
from __future__ import annotations

import itertools
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "general_code_b200" / "csrc"

SOURCE = r"""
#include "gc_offaxis_tree.h"
#include <cstdio>
using namespace gc;
int main() {
  int n, per_chunk, levels, L[3] = {6, 5, 4};
  if (std::scanf("%d %d %d", &n, &per_chunk, &levels) != 3)
    return 1;
  std::vector<OffaxisLine> lines(n);
  for (auto &l : lines) {
    int m;
    if (std::scanf("%d", &m) != 1)
      return 1;
    l.pattern.resize(m);
    for (int &e : l.pattern)
      if (std::scanf("%d", &e) != 1)
        return 1;
  }
  const OffaxisTree t = offaxis_tree(L, lines, per_chunk, levels);
  auto row = [](const char *name, const std::vector<int> &v) {
    std::printf("%s", name);
    for (int x : v)
      std::printf(" %d", x);
    std::printf("\n");
  };
  row("distinct", t.distinct);
  row("first", t.first);
  row("chunk_nodes", t.chunk_nodes);
  row("chunk_lines", t.chunk_lines);
  for (const OffaxisNode &q : t.nodes)
    std::printf("node %d %d %d %d %d %d %d %d\n", q.d[0], q.d[1], q.d[2], q.line, q.axis,
                q.back, q.from, q.push);
}
"""


@pytest.fixture(scope="module")
def tree(tmp_path_factory):
    d = tmp_path_factory.mktemp("tree")
    (d / "tree.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), str(d / "tree.cpp"), "-o",
                    str(d / "tree")], check=True)

    def run(lines, per_chunk, levels):
        text = f"{len(lines)} {per_chunk} {levels}\n" + "\n".join(
            " ".join(map(str, (len(p),) + p)) for p in lines)
        out = {"node": []}
        for row in subprocess.run([str(d / "tree")], input=text, capture_output=True, text=True,
                                  check=True).stdout.splitlines():
            name, *vals = row.split()
            vals = [int(v) for v in vals]
            if name == "node":
                out["node"].append(vals)
            else:
                out[name] = vals
        return out
    return run


def _lines(n, seed):
    rng = random.Random(seed)
    steps = [1, 2, 3, -1, -2, -3]
    lines = [tuple(rng.choice(steps) for _ in range(rng.randint(1, 7))) for _ in range(n)]
    return lines + lines[: n // 3]  # (some twice)


def _complete(t, lines, per_chunk):
    distinct = len(set(lines))
    assert len(t["first"]) == distinct and len(t["distinct"]) == len(lines)
    assert [lines[t["first"][d]] for d in t["distinct"]] == lines
    cl = t["chunk_lines"]
    assert cl[0] == 0 and cl[-1] == distinct
    assert all(0 < b - a <= per_chunk for a, b in itertools.pairwise(cl))


@pytest.mark.parametrize("per_chunk", [1, 5, 48])
def test_walk_gives_every_line(tree, per_chunk):
    lines = _lines(90, per_chunk)
    t = tree(lines, per_chunk, 12)
    _complete(t, lines, per_chunk)
    assert len(t["chunk_nodes"]) == len(t["chunk_lines"]) and t["chunk_nodes"][-1] == len(t["node"])
    found = {}
    for n0, n1 in itertools.pairwise(t["chunk_nodes"]):
        stack, product = {}, None
        for *d, line, axis, back, src, push in t["node"][n0:n1]:
            before = () if src == -2 else product if src == -1 else stack[src]
            product = before + ((-1 if back else 1) * (axis + 1),)
            at = [0, 0, 0]
            for e in product[:-1]:
                at[abs(e) - 1] += 1 if e > 0 else -1
            at[axis] -= back
            assert d == [a % L for a, L in zip(at, (6, 5, 4))]
            if push >= 0:
                stack[push] = product
            if line >= 0:
                found[line] = product
    assert found == {k: lines[i] for k, i in enumerate(t["first"])}


@pytest.mark.parametrize("levels", [-1, 0, 1])
def test_lines_and_chunks_are_complete_without_room_on_the_stack(tree, levels):
    lines = _lines(90, 7)
    t = tree(lines, 30, levels)
    assert t["node"] == []
    _complete(t, lines, 30)
