"""The axis tables of the one-launch FP64 contraction, compiled for the host:
every entry against the offset it stands for, and beyond the limit a refusal
that leaves the tables as they were (the step then takes the packed path)."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

CHECK = r"""
#include <cstdio>
#include "contract_f64.hpp"
using Legs = std::vector<std::pair<int64_t, int64_t>>;
static int check(tnx::AxisTabs& T, const Legs& legs) {
  int32_t t = -7, str = -7;
  if (!T.add(legs, &t, &str)) return 2;
  int64_t n = 1;
  for (auto& l : legs) n *= l.first;
  for (int64_t i = 0; i < n; ++i) {
    int64_t rem = i, off = 0;
    for (size_t l = legs.size(); l-- > 0;) off += (rem % legs[l].first) * legs[l].second, rem /= legs[l].first;
    if (off != (t < 0 ? i * str : T.tab[t + i])) return 1;
  }
  return 0;
}
int main() {
  tnx::AxisTabs T;
  T.limit = 100;
  int bad = 0;
  bad += check(T, {}) != 0;                                   // no leg
  bad += check(T, {{1, 5}, {7, 3}}) != 0;                     // one leg that counts
  bad += check(T, {{5, 12}, {4, 3}}) != 0 || !T.tab.empty();  // merges: a stride, no table
  bad += check(T, {{5, 3}, {4, 20}}) != 0 || T.tab.size() != 20;
  bad += check(T, {{5, 3}, {1, 9}, {4, 20}}) != 0 || T.tab.size() != 20;  // the same legs: the same table
  bad += check(T, {{9, 3}, {9, 40}}) != 2 || T.tab.size() != 20;          // 20 + 81 entries: refused
  bad += check(T, {{8, 3}, {10, 40}}) != 0 || T.tab.size() != 100;        // 20 + 80: filled
  bad += check(T, {{2, 3}, {2, 50}}) != 2 || T.tab.size() != 100;
  int32_t t, str;
  tnx::AxisTabs D;  // far beyond any limit: refused at once, not filled first
  bad += D.add({{1 << 20, 3}, {1 << 20, 4 << 20}}, &t, &str) || !D.tab.empty();
  tnx::AxisTabs E;
  bad += check(E, {{3, 1000}, {5, 7}, {4, 90}, {2, 1}}) != 0 || E.tab.size() != 120;
  bad += check(E, {{3, 7}, {0, 5}}) != 0 || E.tab.size() != 120;  // an empty axis
  return bad;
}
"""


# the longest K span and the most rows whose offsets inside a tile fit 32 bits
LIMITS = r"""
#include "contract_f64.hpp"
static int64_t most(int64_t deep, int64_t stride) {  // steps of `stride` from 0 that end below 2^31, at most `deep`
  int64_t n = 1;
  while (n < deep && n * stride <= INT32_MAX) ++n;
  return n;
}
int main() {
  int bad = 0;
  for (int64_t s : {int64_t{0}, int64_t{1}, int64_t{1} << 24, int64_t{INT32_MAX} / 127, int64_t{INT32_MAX} / 127 + 1,
                    int64_t{INT32_MAX} / 15, int64_t{INT32_MAX} / 15 + 1, int64_t{1} << 30, int64_t{INT32_MAX},
                    int64_t{INT32_MAX} + 1, int64_t{1} << 40}) {
    const int64_t k = tnx::span_k(5000, s), m = tnx::matrix_rows(5000, s);
    bad += k != (most(16, s) == 16 ? 5000 : most(16, s));
    bad += m != (most(128, s) == 128 ? 5000 : most(128, s));
  }
  return bad;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.isdir(os.path.join(CUDA, "include")),
                    reason="needs g++ and the CUDA headers")
@pytest.mark.parametrize("code", [CHECK, LIMITS], ids=["tables", "limits"])
def test_axis_tables(tmp_path, code):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(code)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{os.path.join(ROOT, 'tenax_b200', 'csrc')}",
                    f"-I{os.path.join(CUDA, 'include')}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
