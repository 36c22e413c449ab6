"""Host check of the smooth union's cell masks and blend (csrc/ar_sdf.h).

A march evaluates the union over the primitives its cell lists (sdf_cell_mask).
That must return what the plain left fold over all primitives returns, bit for
bit, at every point of the cell: checked on random unions (sizes, widths, far
from the origin, more than 32 primitives) at random points of a grid built as
the GPU builds it, many near cell borders.  sdf_over_k must equal the IEEE
quotient for every width and 0 <= x <= k."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "aperturerendererv3_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include <vector_types.h>
#include "ar_sdf.h"
using namespace ar;

static float plain_fold(const std::vector<float4>& pr, int n, float k, V3 p)
{
    float d = sdf_prim(pr[0], pr[1], p);
    for (int i = 1; i < n; ++i) d = smin_poly(d, sdf_prim(pr[2 * i], pr[2 * i + 1], p), k);
    return d;
}

static bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0; }

int main()
{
    std::mt19937 rng(99);
    std::uniform_real_distribution<float> U(0.0f, 1.0f);
    long long checked = 0, bad = 0, masked = 0, all = 0;
    for (int scene = 0; scene < 60; ++scene)
    {
        const int n = 1 + (int)(U(rng) * 64) % 64;
        const float k = (scene % 3 == 0) ? 0.001f + 0.01f * U(rng) : 0.02f + 0.2f * U(rng);
        const float off = (scene % 4 == 0) ? 100.0f * U(rng) : 0.0f;
        std::vector<float4> pr(2 * n);
        SdfUnion s;
        s.lo = v3(3e38f, 3e38f, 3e38f);
        s.hi = v3(-3e38f, -3e38f, -3e38f);
        for (int i = 0; i < n; ++i)
        {
            float4 a, b;
            a.x = (float)((int)(U(rng) * 3) % 3);
            a.y = off + U(rng);
            a.z = off + 0.4f * U(rng);
            a.w = U(rng);
            b.x = 0.02f + 0.2f * U(rng);
            b.y = 0.01f + 0.1f * U(rng);
            b.z = 0.02f + 0.2f * U(rng);
            b.w = sdf_bounding_radius(a.x, b.x, b.y, b.z);
            pr[2 * i] = a;
            pr[2 * i + 1] = b;
            const float r = b.w + 0.25f * k;
            s.lo = vmin(s.lo, v3(a.y - r, a.z - r, a.w - r));
            s.hi = vmax(s.hi, v3(a.y + r, a.z + r, a.w + r));
        }
        s.prims = pr.data();
        s.count = n;
        s.k = k;
        s.rk = sdf_reciprocal_k(k);
        const int res = 8 + scene % 25;
        const V3 ext = s.hi - s.lo;
        const V3 cell = v3(ext.x / res, ext.y / res, ext.z / res);
        std::vector<unsigned long long> cells((size_t)res * res * res);
        for (int z = 0; z < res; ++z)
            for (int y = 0; y < res; ++y)
                for (int x = 0; x < res; ++x)
                {
                    const V3 c = s.lo + v3(((float)x + 0.5f) * cell.x, ((float)y + 0.5f) * cell.y, ((float)z + 0.5f) * cell.z);
                    cells[((size_t)z * res + y) * res + x] = sdf_cell_mask(s, c, 0.5f * length(cell) * 1.001f);
                }
        s.res[0] = s.res[1] = s.res[2] = res;
        s.inv_cell = v3(1.0f / cell.x, 1.0f / cell.y, 1.0f / cell.z);
        s.cells = cells.data();
        for (int j = 0; j < 20000; ++j)
        {
            V3 u = v3(U(rng), U(rng), U(rng));
            if (j % 3 == 0)  // near the cells' borders
                u = v3(std::round(u.x * res) / res + 1e-6f * (U(rng) - 0.5f), std::round(u.y * res) / res, u.z);
            const V3 p = s.lo + v3(u.x * ext.x, u.y * ext.y, u.z * ext.z);
            if (!same(sdf_union(s, p), plain_fold(pr, n, k, p))) ++bad;
            masked += __builtin_popcountll(sdf_mask(s, p));
            all += n;
            ++checked;
        }
    }
    long long qbad = 0, qn = 0;
    for (int t = 0; t < 4000; ++t)
    {
        float k = std::ldexp(0.5f + 0.5f * U(rng), (int)(U(rng) * 40) - 20);
        if (t % 50 == 0) k = std::nextafter(std::ldexp(1.0f, t % 7), 0.0f);  // a significand of ones
        const float rk = sdf_reciprocal_k(k);
        for (int j = 0; j < 500; ++j)
        {
            float x = k * U(rng);
            if (j % 5 == 0) x = k - k * std::ldexp(U(rng), -20);
            if (j == 1) x = k;
            if (j == 2) x = 0.0f;
            if (j == 3) x = std::ldexp(k, -24);
            ++qn;
            if (!same(sdf_over_k(x, k, rk), x / k)) ++qbad;
        }
    }
    std::printf("%lld %lld %lld %lld %lld %lld\n", checked, bad, masked, all, qn, qbad);
    return 0;
}
"""


def test_cell_masks_equal_the_plain_fold(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    cuda_inc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    if not (cuda_inc / "vector_types.h").exists():
        pytest.skip("CUDA headers (vector types) not found")
    src = tmp_path / "cells.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "cells"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), "-I", str(cuda_inc), str(src),
                    "-o", str(exe)], check=True)
    checked, bad, masked, total, qn, qbad = map(
        int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert checked == 60 * 20000 and bad == 0
    assert masked < 0.7 * total  # the masks do leave primitives out
    assert qn == 4000 * 500 and qbad == 0
