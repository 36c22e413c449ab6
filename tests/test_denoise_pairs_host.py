"""Host check of the denoiser's quick pair test (csrc/ar_denoise_test.h).

dn_channel_quick and dn_channel_nu decide most t-tests without divisions and the
square root; they must never contradict dn_channel_passes, the reference's
arithmetic, and leave few pairs undecided.  Checked on random moments over many orders of magnitude,
pairs placed at both thresholds and within a few ulp of them, equal and
different sample counts inside a tile's range, and zero, infinite and undefined
values."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "aperturerendererv3_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "ar_denoise_test.h"
#include "ar_t_quantile.h"
using namespace ar;

int main()
{
    std::mt19937 rng(7);
    std::uniform_real_distribution<float> U(0.0f, 1.0f);
    std::vector<float> tq(ar_t_quantile_0025, ar_t_quantile_0025 + kDnQuantiles), k2(kDnQuantiles);
    for (int i = 0; i < kDnQuantiles; ++i) k2[i] = 2.0f * (1.0f + tq[i] * tq[i]);
    long long n = 0, wrong = 0, undecided = 0, undecided2 = 0, random_n = 0, passes = 0;
    const float special[] = {0.0f, -0.0f, 1e-45f, 1e-38f, 1e-20f, 1e-7f, 1.0f, 1e20f, 3e38f, INFINITY, -INFINITY, NAN, -1.0f};
    for (int it = 0; it < 6000000; ++it)
    {
        const int mode = it % 4;
        const float scale = std::ldexp(1.0f, (int)(U(rng) * 60) - 40);
        // two pixels of a tile: their sample counts, variances of theta and Welch terms
        const uint32_t fA = 1 + (uint32_t)(U(rng) * (it % 3 ? 40 : 3000)), fB = it % 5 ? fA : 1 + (uint32_t)(U(rng) * 400);
        const uint32_t f0 = std::min(fA, fB), f1 = std::max(fA, fB) + (it % 7 == 0 ? 20 : 0);
        float vA = scale * (0.05f + U(rng)), vB = scale * (0.05f + U(rng)), t = std::sqrt(scale) * 8.0f * (U(rng) - 0.5f);
        if (mode == 2) { vB = vA; if (it % 8 == 2) t = 0.0f; }
        if (mode == 3)
        {
            float* f[3] = {&t, &vA, &vB};
            for (int k = 0; k < 1 + (it % 3); ++k) *f[(int)(U(rng) * 3) % 3] = special[(int)(U(rng) * 13) % 13];
        }
        const float u = vA + vB, lo = vA * vA / (float)fA + vB * vB / (float)fB;
        if (mode == 1)
        {
            // at a threshold: t^2 + vB = vA, or rho = 2 (1 + q^2)
            const float q = dn_t_quantile(tq.data(), u * u / lo);
            const double target = (it % 8 < 4) ? (double)vA - vB : 2.0 * vA * (1.0 + (double)q * q) - vA - vB;
            if (target > 0) t = (float)std::sqrt(target);
            const int steps = (int)(U(rng) * 9) - 4;
            for (int s = 0; s < std::abs(steps); ++s) t = std::nextafter(t, steps > 0 ? 3e38f : 0.0f);
        }
        const bool ex = dn_channel_passes(t, vA, vB, u, lo, tq.data());
        bool pass, fail;
        dn_channel_quick(t, vA, 1.0f / vA, vB, dn_rho_limits(f0, f1, tq.data()), &pass, &fail);
        if (!dn_ordinary(vA, vA) || !dn_ordinary(vB, vB)) continue;  // such tiles take dn_channel_passes
        ++n;
        passes += ex;
        if ((pass && !ex) || (fail && ex) || (pass && fail)) ++wrong;
        if (mode == 0 && it % 5 && it % 7) { ++random_n; undecided += !pass && !fail; }
        dn_channel_nu(t, vA, 1.0f / vA, vB, lo, k2.data(), &pass, &fail);
        if ((pass && !ex) || (fail && ex) || (pass && fail)) ++wrong;
        if (mode == 0 && it % 5 && it % 7) undecided2 += !pass && !fail;
    }
    std::printf("%lld %lld %lld %lld %lld %lld\n", n, wrong, random_n, undecided, undecided2, passes);
    return 0;
}
"""


def test_quick_test_never_contradicts_the_reference_arithmetic(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = tmp_path / "pairs.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "pairs"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    n, wrong, random_n, undecided, undecided2, passes = map(
        int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert n > 5_000_000 and passes > n // 20
    assert wrong == 0
    # equal sample counts: only a rho between the quantiles of f and 2 f, or tiny variances, stay open
    assert undecided < 0.4 * random_n
    # with the pair's own degrees of freedom: tiny variances (a third of the magnitudes drawn), thresholds
    assert undecided2 < 0.4 * random_n
