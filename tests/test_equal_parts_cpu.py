"""Equal parts of a launch's edges, with the kernels' own arithmetic compiled for the host and the searches in the row table
restated: every edge is in one part, every row is ended by one team, and no index into the row table lies outside it.  The last
is out of a kernel test's sight: what a part without rows reads there changes no result."""

import os
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lunaequivariance_b200", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "uvu_parts.cuh"
using namespace luna::edgek;

static const char* what = "";
[[noreturn]] void fail(const char* why, long a, long b) {
  std::printf("%s: %s (%ld, %ld)\n", what, why, a, b);
  std::exit(1);
}
struct RowTable {  // rows + 1 entries
  std::vector<int> entries;
  int rows() const { return static_cast<int>(entries.size()) - 1; }
  int operator[](int at) const {
    if (at < 0 || at > rows()) fail("index outside the row table, entries", at, rows() + 1);
    return entries[at];
  }
};
RowTable table(const std::vector<int>& degrees) {
  RowTable t{{0}};
  for (int d : degrees) t.entries.push_back(t.entries.back() + d);
  return t;
}
// as team_part (uvu_edge.cuh), whose warps search the row table
struct FoundRow {
  int row, begin;
};
TeamPart cut(const RowTable& t, int block, int blocks, int team, int teams) {
  auto find = [&](long bound) {
    const int row = static_cast<int>(std::lower_bound(t.entries.begin(), t.entries.end(), bound) - t.entries.begin());
    return FoundRow{row, t[row]};
  };
  const long edges = t.entries.back();
  const FoundRow from = find(edges * block / blocks);
  const FoundRow to = block + 1 == blocks ? FoundRow{t.rows(), static_cast<int>(edges)} : find(edges * (block + 1) / blocks);
  TeamPart p;
  p.cta_pos = from.begin;
  p.cta_edges = to.begin - from.begin;
  p.pos = part_begin(p.cta_pos, p.cta_edges, team, teams);
  p.end = part_begin(p.cta_pos, p.cta_edges, team + 1, teams);
  const FoundRow first = find(p.pos), last = find(p.end);
  p.n = first.row;
  p.n_hi = team + 1 == teams ? to.row : last.row;
  p.joined = p.pos < p.end && first.begin > p.pos;
  p.open = team + 1 < teams && p.pos < p.end && last.begin > p.end;
  if (p.joined) --p.n;
  return p;
}
void check(const RowTable& t, int blocks, int teams, const char* name) {
  what = name;
  const int rows = t.rows(), edges = t.entries.back();
  std::vector<char> edge(edges, 0), ended(rows, 0);
  for (int block = 0; block < blocks; ++block) {
    int open = -1;
    for (int team = 0; team < teams; ++team) {
      const TeamPart p = cut(t, block, blocks, team, teams);
      if (p.n < 0 || p.n_hi > rows || p.end > edges) fail("part outside the graph", p.n, p.n_hi);
      for (int e = p.pos; e < p.end; ++e)
        if (edge[e]++) fail("edge taken twice", e, team);
      // as the forward of two edges at a time walks the rows
      int n = p.n, row_end = first_row_end(t, n, p.n_hi, p.end);
      for (int e = p.pos; e < p.end; ++e) {
        while (e >= row_end) row_end = std::min(t[++n + 1], p.end);
        if (e < t[n] || e >= t[n + 1]) fail("edge of another row", e, n);
      }
      if (p.joined && open != p.n) fail("joined a row that is not open", p.n, open);
      if (p.pos < p.end) open = p.open_row();
      for (n = p.n; n < p.n_hi; ++n)
        if (n != p.open_row() && ended[n]++) fail("row ended twice", n, team);
      if (p.closes() && t[p.n] >= p.pos) fail("closes a row that began here", p.n, team);
    }
    if (open != -1) fail("row left open", open, block);
  }
  for (int e = 0; e < edges; ++e)
    if (!edge[e]) fail("edge left out", e, edges);
  for (int n = 0; n < rows; ++n)
    if (!ended[n]) fail("row left out", n, rows);
}

int main() {
  auto repeat = [](int count, int degree) { return std::vector<int>(count, degree); };
  auto with = [](std::vector<int> degrees, const std::vector<int>& more) {
    degrees.insert(degrees.end(), more.begin(), more.end());
    return degrees;
  };
  for (int teams : {1, 2, 7, 16, 24})
    for (int sms : {148, 132, 5}) {
      auto all = [&](const RowTable& t, const char* name) { check(t, std::max(1, std::min(sms, t.rows())), teams, name); };
      all(table(repeat(500, 4)), "500 rows of 4");
      all(table(repeat(450, 5)), "450 rows of 5");
      all(table(with(repeat(1000, 16), {200})), "1000 rows of 16 and a long last one");
      all(table(with(repeat(1000, 20), {900, 0, 0})), "a long row and two empty ones at the end");
      all(table(with({0, 0, 700}, repeat(600, 4))), "empty rows and a long one first");
      all(table({1}), "one edge");
      all(table({0, 3000, 0}), "one row has all edges");
      std::mt19937 generator(7);
      for (int i = 0; i < 60; ++i) {
        std::vector<int> degrees(1 + generator() % 900);
        for (int& d : degrees) d = generator() % 4 ? generator() % 12 : generator() % (i % 3 ? 3 : 200);
        degrees[generator() % degrees.size()] += 1;
        all(table(degrees), "random rows");
      }
    }
  return 0;
}
"""


def test_every_edge_and_row_once_and_no_index_outside_the_row_table(tmp_path):
    source, program = tmp_path / "parts.cpp", tmp_path / "parts"
    source.write_text(PROGRAM)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", f"-I{CSRC}", "-x", "c++", str(source), "-o", str(program)],
                   check=True)
    result = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert result.returncode == 0, result.stdout
