"""The CUDA sources that set up tensor maps through pq_tc.cuh pass nvcc's front end without a warning (a warning there is a declaration that it had to change, such
as a function-local `inline` variable, which became one per call)."""
import concurrent.futures as cf
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_front_end_is_silent(tmp_path):
    from polyquant_gb300 import build

    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")

    def run(src):
        out = tmp_path / (os.path.basename(src) + ".ii")
        r = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", build.CSRC,
                            "-Werror", "all-warnings", "--cuda", "-o", str(out), src], capture_output=True, text=True)
        return "" if r.returncode == 0 else f"{os.path.basename(src)}: {r.stdout}{r.stderr}"

    def maps(src):
        with open(src) as f:
            text = f.read()
        return "pq_tc.cuh" in text or "ci_dense64.cuh" in text

    srcs = [s for s in build.sources() if s.endswith(".cu") and maps(s)]
    assert len(srcs) >= 3
    with cf.ThreadPoolExecutor(max_workers=4) as ex:
        bad = [m for m in ex.map(run, srcs) if m]
    assert not bad, "\n".join(bad)
