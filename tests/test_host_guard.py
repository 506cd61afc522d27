"""A host allocation that fails inside a sigma, a solve, an explicit build or a property call comes back as PQ_ERR_OOM
instead of leaving the C entry as an exception, and is tried again once the handle's optional tables are gone."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SRC = r"""
#include <cstdio>
#include "pq_internal.h"
static int drops = 0, errors = 0, left = 0;
namespace pq {
void set_error(const char *, ...) { errors++; }
void clear_error() {}
bool ci_drop_tables(pq_ci_handle *) { drops++; return left-- > 0; }
}
int main() {
  using namespace pq;
  auto bad = []() -> pq_status { throw std::bad_alloc(); };
  if (host_guard(bad) != PQ_ERR_OOM || errors != 1) return 1;
  if (host_guard([] { return (pq_status)PQ_ERR_ARG; }) != PQ_ERR_ARG) return 2;
  if (with_room(nullptr, bad) != PQ_ERR_OOM || drops != 1) return 3;
  left = 2, drops = 0;
  int calls = 0;
  if (with_room(nullptr, [&]() -> pq_status {
        if (++calls < 3) throw std::bad_alloc();
        return PQ_OK;
      }) != PQ_OK || calls != 3 || drops != 2) return 4;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(os.path.join(CUDA, "include")),
                    reason="no host compiler or CUDA headers")
def test_failed_host_allocation_is_a_status(tmp_path):
    src = tmp_path / "guard.cpp"
    src.write_text(SRC)
    obj = tmp_path / "guard.o"
    inc = ["-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "polyquant_gb300", "csrc"), "-I", os.path.join(CUDA, "include")]
    r = subprocess.run(["g++", "-std=c++17", "-O1", *inc, "-c", str(src), "-o", str(obj)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run(["g++", str(obj), "-o", str(tmp_path / "guard"), "-Wl,--gc-sections"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(tmp_path / "guard")]).returncode == 0
