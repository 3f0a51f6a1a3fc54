"""Which meshes the keyed finite-depth fill takes (hg_fin_keys.cuh, on the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include "hg_fin_keys.cuh"
int main(int c, char** v) {
  std::printf("%d\n", (int)hg::keys_index(atoi(v[1]), atoi(v[2]), atoi(v[3]), atoi(v[4])));
  return 0;
}
'''


@pytest.fixture(scope="module")
def index(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("keys")
    src, exe = d / "keys.cpp", d / "keys"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-w", "-I", os.path.join(ROOT, "hams-mrel_gb300", "csrc"), "-I",
                    os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)
    return lambda *a: subprocess.run([str(exe), *map(str, a)], check=True, capture_output=True, text=True).stdout == "1\n"


# all pairs up to 2^27; near pairs of any mesh whose pair index fits an int (12096 panels and more); 2^18 depths
@pytest.mark.parametrize("tn,n,near,nlev,want", [(11585, 11585, 0, 100, True), (11586, 11586, 0, 100, False),
                                                 (12096, 12096, 1, 100, True), (46340, 46340, 1, 100, True),
                                                 (46341, 46341, 1, 100, False), (20000, 6000, 1, 1 << 18, True),
                                                 (20000, 6000, 0, (1 << 18) + 1, False)])
def test_pairs_that_can_be_keyed(index, tn, n, near, nlev, want):
    assert index(tn, n, near, nlev) == want
