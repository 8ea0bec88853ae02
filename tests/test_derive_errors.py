"""Derived arrays of an index on a host without a GPU: an allocation that fails for another reason
than memory ends the build, and does not read as "no room" for an optional array."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "index.h"
int main(int, char** argv) {
  lshg::Index I;
  I.p.implementation = 2;
  I.n = 5000;
  I.d = 100;
  I.C = 1024;
  I.dist = 1;
  try {
    if (argv[1][0] == 'e') lshg::derive_exact(I, nullptr);
    if (argv[1][0] == 'j') I.dist = 2, lshg::derive_jaccard_scan(I, nullptr);
    if (argv[1][0] == 'r') I.sk_kind = 3, lshg::derive_rerank_bounds(I, nullptr);
  } catch (const lshg::Error& e) {
    std::printf("%d", e.status);
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(engine, tmp_path_factory):
    import torch

    from lshongpu_gb300 import build

    if torch.cuda.is_available():
        pytest.skip("allocations succeed where there is a GPU")
    td = tmp_path_factory.mktemp("derive")
    src, exe = str(td / "derive.cu"), str(td / "derive")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-cudart", "shared", "-o", exe, src, "-L" + build.LIBDIR,
                    "-llshg", "-Xlinker", "-rpath=" + build.LIBDIR], check=True)
    return exe


@pytest.mark.parametrize("what", ["exact", "jaccard", "rerank"])
def test_derive_reports_errors_other_than_memory(program, what):
    out = subprocess.run([program, what], capture_output=True, text=True, check=True).stdout
    assert out == "2", f"status {out or 'none'} instead of LSHG_ERR_CUDA"
