"""The key under which an ensemble's captured launch sequence is replayed
(csrc/clmd_ens_launch.hpp), on the host alone: two launches that differ in
anything a captured kernel argument or launch attribute is made from have
different keys."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "fortran-cluster-md_b200", "csrc")

DRIVER = r"""
#include "clmd_ens_launch.hpp"
#include <cstdio>
#include <cstring>

static ClassLaunch base(int item0, int nitems) {
  ClassLaunch a;
  a.k = (EnsKernel)0x1000;
  a.smem = 90112; a.grid = 148; a.nt = 1024;
  a.item0 = item0; a.nitems = nitems;
  return a;
}

int main(int, char** v) {
  // 300 replicas in two classes that both fill the GPU: 160 + 140
  int items[300];
  for (int k = 0; k < 300; k++) items[k] = k;
  ClassLaunch a[2] = {base(0, 160), base(160, 140)}, b[2] = {a[0], a[1]};
  int nwin = 1;
  bool balanced = false;
  if (!strcmp(v[1], "split")) {  // the last of class 0 now the first of class 1
    b[0] = base(0, 159); b[1] = base(159, 141);
  } else if (!strcmp(v[1], "cs")) { b[1].cs = 4;
  } else if (!strcmp(v[1], "lg")) { b[1].lg = 1;
  } else if (!strcmp(v[1], "region")) { b[1].region0 = 8;
  } else if (!strcmp(v[1], "grid")) { b[1].grid = 147;
  } else if (!strcmp(v[1], "smem")) { b[1].smem += 8;
  } else if (!strcmp(v[1], "threads")) { b[1].nt = 512;
  } else if (!strcmp(v[1], "kernel")) { b[1].k = (EnsKernel)0x2000;
  } else if (!strcmp(v[1], "windows")) { nwin = 2;
  } else if (!strcmp(v[1], "balanced")) { balanced = true;
  }
  const auto ka = launch_key(1, false, items, 300, a, 2);
  if (!strcmp(v[1], "order")) { items[3] = 4; items[4] = 3; }
  puts(ka == launch_key(nwin, balanced, items, 300, b, 2) ? "equal" : "different");
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("key")
    (d / "key.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(d / "key.cpp"), "-o", str(d / "key")],
                   check=True, capture_output=True)
    return str(d / "key")


@pytest.mark.parametrize("change", ["split", "cs", "lg", "region", "grid", "smem", "threads",
                                    "kernel", "windows", "balanced", "order", "none"])
def test_launch_key(driver, change):
    out = subprocess.run([driver, change], capture_output=True, text=True, check=True).stdout
    assert out.strip() == ("equal" if change == "none" else "different")
