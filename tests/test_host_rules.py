"""Rules that the library's host code goes by, called from a small C++ program
(no GPU: they are plain functions of sizes and attributes)."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "caps-sa_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "common.cuh"
using namespace capssa;

int main() {
    // reach: memory type, its device, the context's device -> read in place?
    const cudaMemoryType types[] = {cudaMemoryTypeUnregistered, cudaMemoryTypeHost,
                                    cudaMemoryTypeDevice, cudaMemoryTypeManaged};
    std::printf("{\"reach\": [");
    for (int t = 0; t < 4; t++)
        for (int d = 0; d < 3; d++)
            for (int c = 0; c < 3; c++) {
                cudaPointerAttributes a{};
                a.type = types[t];
                a.device = d;
                std::printf("%s[%d, %d, %d, %d]", t || d || c ? ", " : "", t, d, c,
                            (int)kernels_reach(a, c));
            }
    std::printf("]}\n");
    return 0;
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "caps-sa_gb300"))
    import build
    d = tmp_path_factory.mktemp("rules")
    src, exe = str(d / "rules.cu"), str(d / "rules")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", CSRC, src, "-o", exe],
                   check=True, capture_output=True, text=True)
    return json.loads(subprocess.run([exe], check=True, capture_output=True, text=True).stdout)


def test_a_text_is_read_in_place_on_its_own_gpu_only(rules):
    """Host memory never, device memory on the context's GPU, managed memory
    anywhere; everything else is copied first."""
    assert len(rules["reach"]) == 36
    for kind, device, context, reach in rules["reach"]:
        want = kind == 3 or (kind == 2 and device == context)
        assert bool(reach) == want, (kind, device, context)
