"""The division of a ray batch among warps (csrc/ar_ray_share.h): every ray of a batch
has exactly one place, for batches up to the largest int."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "aperturerendererv3_gb300" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include "ar_ray_share.h"
using namespace ar;

int main(int argc, char** argv)
{
    const long long n = std::atoll(argv[1]);
    const RayShare s{(int)n, std::atoi(argv[2]), std::atoi(argv[3])};
    const int chunk = 1 << s.chunk_log2;
    long long rays = 0, chunks = 0, bad = 0;
    for (int w = 0; w < s.warps; ++w)
    {
        const int limit = s.limit(w);
        long long last = -1;
        for (int j = 0; j < limit; j += chunk)
        {
            // a chunk's rays follow one another; it is the warp's own and comes after its last one
            const long long r = s.ray(w, j);
            bad += r % chunk != 0 || (r / chunk) % s.warps != w || r <= last || s.ray(w, j + chunk - 1) != r + chunk - 1;
            last = r;
            rays += std::max(0ll, std::min((long long)chunk, n - r));
            ++chunks;
        }
    }
    std::printf("%lld %lld %lld\n", rays, chunks - s.chunks(), bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    if not nvcc.exists():
        nvcc = shutil.which("nvcc")
        if nvcc is None:
            pytest.skip("nvcc not found")
    tmp = tmp_path_factory.mktemp("share")
    src, exe = tmp / "share.cu", tmp / "share"
    src.write_text(PROGRAM)
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("n,chunk_log2,warps", [
    (1, 0, 4), (2432, 0, 2432), (2433, 0, 2436), (4865, 1, 2436), (77825, 5, 2436), (2073600, 5, 4864),
    (2**31 - 33, 5, 4864), (2**31 - 32, 5, 4864), (2**31 - 31, 5, 4864), (2**31 - 1, 5, 4864), (2**31 - 1, 5, 4736)])
def test_every_ray_has_one_place(program, n, chunk_log2, warps):
    out = subprocess.run([str(program), str(n), str(chunk_log2), str(warps)], check=True, capture_output=True,
                         text=True).stdout.split()
    assert [int(v) for v in out] == [n, 0, 0]
