// tn_workspace.h -- device scratch of an executor launch: a workspace per CTA,
// and beside it the parts that bond_team needs (one per CTA or cluster), taken
// when a launch with wide bonds first asks for them.  Host logic only; the
// allocator is a parameter.
//
// Memory decides how many parts there are, never whether a launch is correct:
// without a part a CTA runs the block Jacobi on the base workspace, and only a
// launch that has a part for every cluster uses clusters (launch_shape).
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace tn {

// Mem: int alloc(void **, size_t) (0: done), void free(void *), size_t available().
template <class Mem>
struct Workspace {
  Mem mem;
  size_t stride = 0, team_stride = 0;  // bytes of a CTA's workspace and of a part (0: no parts here)
  bool keep_parts = false;  // parts that were replaced stay until release(): captured launches point to them
  void *base = nullptr, *team = nullptr;
  int ctas = 0, teams = 0;
  std::vector<void *> former;

  Workspace() = default;
  Workspace(const Workspace &) = delete;
  Workspace &operator=(const Workspace &) = delete;
  ~Workspace() { release(); }

  void release() {
    if (base) mem.free(base);
    if (team) mem.free(team);
    for (void *p : former) mem.free(p);
    base = team = nullptr;
    ctas = teams = 0;
    former.clear();
  }

  // At least n workspaces.  The present ones stay until the new ones are there;
  // when memory does not hold both they go first, and come back if even that is
  // too little.  Nothing may be running on them when n grows.
  int ensure(int n) {
    if (n <= ctas) return 0;
    void *p = nullptr;
    int e = mem.alloc(&p, stride * size_t(n));
    if (e && base) {
      const int had = ctas;
      mem.free(base);
      base = nullptr;
      ctas = 0;
      e = mem.alloc(&p, stride * size_t(n));
      if (e) {
        if (mem.alloc(&base, stride * size_t(had)) == 0)
          ctas = had;
        else
          base = nullptr;
        return e;
      }
    }
    if (e) return e;
    if (base) mem.free(base);
    base = p;
    ctas = n;
    return 0;
  }

  // Parts for `want` CTAs or clusters, or for half of them, a quarter, ... down
  // to `least`, in at most half of the memory that is free (what a program
  // allocates next finds room as it did without them).  Returns how many there
  // are; 0: none.  Nothing may be running on the present ones unless they are kept.
  int ensure_teams(int want, int least = 1) {
    if (team_stride == 0 || want <= teams) return teams;
    const size_t room = mem.available() / 2;
    for (int n = want; n >= std::max(least, teams + 1); n = n > 1 ? (n + 1) / 2 : 0) {
      void *p = nullptr;
      if (team_stride * size_t(n) <= room && mem.alloc(&p, team_stride * size_t(n)) == 0) {
        if (team && keep_parts)
          former.push_back(team);
        else if (team)
          mem.free(team);
        team = p;
        teams = n;
        break;
      }
    }
    return teams;
  }
};

// Launch of `items` independent operations: CTAs, or clusters of them.
struct LaunchShape {
  bool clusters;  // clusters of CTAs (each has a part)
  int grid;       // CTAs or clusters
  bool parts;     // every one of them has a part
};
// resident: clusters that fit the GPU (0: none); teams: parts that are there.
inline LaunchShape launch_shape(int items, int sms, int resident, int teams) {
  LaunchShape s;
  s.clusters = resident > 0 && teams > 0;
  s.grid = std::max(1, std::min(items, s.clusters ? std::min(resident, teams) : sms));
  s.parts = teams >= s.grid;
  return s;
}

}  // namespace tn
