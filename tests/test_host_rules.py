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
#include "msd.cuh"
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
    // bins: records, ranges, bits asked for -> bits taken
    std::printf("], \"bins\": [");
    const char *sep = "";
    for (unsigned long long n = 5000; n < 1ull << 32; n = n * 3 + 1)
        for (unsigned long long r = 1; r <= n / (msd::kOneBlock / 2 + 1) + 1; r = r * 5 + 2)
            for (int want = 1; want <= msd::kMaxDigit; want++) {
                std::printf("%s[%llu, %llu, %d, %d]", sep, n, r, want, msd::level_bits(n, r, want));
                sep = ", ";
            }
    // pieces: n, at most this many in each -> pieces
    std::printf("], \"pieces\": [");
    sep = "";
    for (unsigned per : {1u, 2560u, 6144u, 8192u})
        for (unsigned n : {1u, 2559u, 2560u, 2561u, 8192u, 8193u, 4294959104u, 4294959105u,
                           4294961152u, 4294964736u, 4294967294u, 4294967295u}) {
            std::printf("%s[%u, %u, %u]", sep, n, per, msd::pieces_of(n, per));
            sep = ", ";
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


def test_bins_of_a_level_stay_within_a_byte_a_record(rules):
    """... or 64 MB; eight bits of digit, what the levels past the planned ones
    take, are never refused, and nothing is cut that fits."""
    assert len(rules["bins"]) > 500
    for n, ranges, want, got in rules["bins"]:
        most = max(n // 4, 1 << 24)
        assert 1 <= got <= want
        assert got >= min(want, 8)
        assert ranges << got <= most
        assert got == want or ranges << (got + 1) > most


def test_pieces_of_the_largest_counts(rules):
    """Up to 2^32 - 1 records: none are lost to a wrapped sum."""
    for n, per, got in rules["pieces"]:
        assert got == -(-n // per)
