"""tn_order.h on the CPU: the ranks that index shared memory are a permutation
for any values (NaN, infinities, equal ones), in decreasing order, and for
finite values the plain decreasing order by index on ties."""
import math
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "tensor-net_gb300" / "csrc"
SOURCE = """
#include <cstdio>
#include <cstdlib>
#include "tn_order.h"
template <typename R> void ranks(int n, char **a) {
  R *v = new R[n];
  for (int i = 0; i < n; ++i) v[i] = R(std::strtod(a[i], nullptr));
  for (int i = 0; i < n; ++i) std::printf("%d ", tn::order_rank(v, n, i));
  std::printf("\\n");
}
int main(int c, char **a) {
  ranks<float>(c - 1, a + 1);
  ranks<double>(c - 1, a + 1);
  double sum = 0;
  for (int i = 1; i < c; ++i) sum += tn::order_square(tn::order_key(std::strtod(a[i], nullptr)));
  std::printf("%d\\n", int(std::isfinite(sum)));
}
"""
NAN, INF = math.nan, math.inf
LISTS = [[1, NAN, .5, .2], [NAN] * 5, [INF, 1, INF, 0], [0, 0, 0], [NAN, INF, -INF, 3, 3, NAN, 1e-30], [2], [NAN],
         [.25, .5, .25, 1, 0], [1, 2, 3, 4, 5, 6, 7, NAN]]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O2", f"-I{CSRC}", str(d / "order.cpp"), "-o", str(d / "order")], check=True)
    return d / "order"


@pytest.mark.parametrize("values", LISTS)
def test_ranks_are_a_permutation(exe, values):
    out = subprocess.run([str(exe), *map(str, values)], capture_output=True, text=True, check=True).stdout.splitlines()
    for line in out[:2]:
        got = [int(x) for x in line.split()]
        assert sorted(got) == list(range(len(values)))
        keys = [v if math.isfinite(v) else -1.0 for v in values]
        assert got == [sorted(range(len(keys)), key=lambda j: (-keys[j], j)).index(j) for j in range(len(keys))]
    assert int(out[2]) == all(math.isfinite(v) for v in values)
