// clmd_ens_launch.hpp -- the launch shape of the ensemble's size classes, and
// the key under which a captured launch sequence may be replayed (host code,
// no CUDA headers).
#pragma once

#include <cstddef>
#include <vector>

namespace clmd_ens {
struct Args;
}
typedef void (*EnsKernel)(clmd_ens::Args);

// the launch shape of one size class: kernel, dynamic shared memory, grid
struct ClassLaunch {
  EnsKernel k = nullptr;
  size_t smem = 0;
  int grid = 0, nt = 0, item0 = 0, nitems = 0;
  int cs = 1;       // CTAs per replica (thread-block cluster size)
  int lg = 0;       // lanes per atom in the mixed force pass: 1 << lg
  int region0 = 0;  // first cell-count region (cluster classes)
};

// Two launches with equal keys are the same sequence: everything that the
// captured kernel arguments and launch attributes are made from is in it.
inline std::vector<long long> launch_key(int nwin, bool balanced, const int* items, int total,
                                         const ClassLaunch* L, int nclass) {
  std::vector<long long> key = {total, nwin, balanced};
  key.insert(key.end(), items, items + total);
  for (int c = 0; c < nclass; c++) {
    // (where the classes fill the GPU, the items' split over them shows in
    // nothing else: not in the items' order, nor in a grid)
    const long long k[] = {(long long)(size_t)L[c].k, (long long)L[c].smem, L[c].grid, L[c].nt,
                           L[c].item0, L[c].nitems, L[c].cs, L[c].lg, L[c].region0};
    key.insert(key.end(), k, k + sizeof(k) / sizeof(k[0]));
  }
  return key;
}
