"""tn_workspace.h on the CPU with an allocator of limited memory: what there is
stays until its replacement is there, refused parts leave a launch without
clusters (never one whose clusters have no part), and parts take at most half
of the free memory."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "tensor-net_gb300" / "csrc"
SOURCE = """
#include <cstdio>
#include <cstdlib>
#include <map>
#include "tn_workspace.h"
static size_t limit, used;
static std::map<void *, size_t> live;
struct Mem {
  int alloc(void **p, size_t n) {
    if (used + n > limit) return 2;
    *p = std::malloc(1);
    live[*p] = n;
    used += n;
    return 0;
  }
  void free(void *p) {
    if (!live.count(p)) std::abort();  // not there, or freed twice
    used -= live[p];
    live.erase(p);
    std::free(p);
  }
  size_t available() { return limit - used; }
};
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\\n", __LINE__, #x); return 1; } } while (0)
int main() {
  {  // growth: both at once where they fit, else the old one first, else the old one again
    tn::Workspace<Mem> w;
    limit = 100;
    w.stride = 10;
    CHECK(w.ensure(2) == 0 && w.ctas == 2 && used == 20);
    void *old = w.base;
    CHECK(w.ensure(1) == 0 && w.base == old);
    CHECK(w.ensure(5) == 0 && w.ctas == 5 && used == 50);
    CHECK(w.ensure(8) == 0 && w.ctas == 8 && used == 80);
    CHECK(w.ensure(11) != 0 && w.ctas == 8 && w.base && used == 80);
    CHECK(w.ensure_teams(4) == 0 && !w.team);  // no parts in this mode
  }
  CHECK(used == 0);
  {  // parts: as many as fit in half of the free memory, by halves
    tn::Workspace<Mem> w;
    limit = 100;
    w.stride = 10;
    w.team_stride = 6;
    CHECK(w.ensure(2) == 0);
    CHECK(w.ensure_teams(16, 16) == 0 && used == 20);  // all or none
    CHECK(w.ensure_teams(16) == 4 && used == 44 && w.team);
    void *had = w.team;
    CHECK(w.ensure_teams(16) == 4 && w.team == had && w.ensure_teams(3) == 4);
    limit = 400;
    CHECK(w.ensure_teams(16) == 16 && w.former.empty() && used == 20 + 96);
    w.keep_parts = true;
    had = w.team;
    CHECK(w.ensure_teams(17) == 17 && w.former.size() == 1 && w.former[0] == had);
  }
  CHECK(used == 0);
  // the launch: clusters only where every one has a part
  for (int items = 1; items < 300; items += 7)
    for (int resident = -1; resident < 40; ++resident)
      for (int teams = 0; teams < 200; teams += 3) {
        const tn::LaunchShape s = tn::launch_shape(items, 152, resident, teams);
        CHECK(s.grid >= 1 && s.grid <= items && s.grid <= 152);
        CHECK(!s.clusters || (s.parts && s.grid <= resident && teams >= s.grid));
        CHECK(s.parts == (teams >= s.grid));
        if (teams == 0 || resident <= 0) CHECK(!s.clusters && s.grid == (items < 152 ? items : 152));
      }
  std::printf("ok\\n");
  return 0;
}
"""


def test_workspace_and_launch_shape_under_memory_pressure(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "ws.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(tmp_path / "ws.cpp"), "-o",
                    str(tmp_path / "ws")], check=True)
    r = subprocess.run([str(tmp_path / "ws")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
