"""The eight lanes of a wide node agree on what they choose together when the GPU
build collapses its tree (csrc/ar_bvh_lanes.h), whatever the children's boxes hold:
lanes that disagreed would drop a child or leave the exchange at different rounds.
The exchanges run here lane by lane, over random boxes with infinite, flat and NaN
ones among them; for finite boxes the winners are those of a serial greedy choice."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "aperturerendererv3_gb300" / "csrc"

PROGRAM = r"""
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <random>
#include "ar_bvh_lanes.h"
using namespace ar::lbvh;

int main()
{
    std::mt19937 rng(8);
    std::uniform_real_distribution<float> U(0.0f, 1.0f);
    long long nodes = 0, unusual = 0, disagree = 0, lost = 0, differ = 0;
    for (int trial = 0; trial < 200000; ++trial)
    {
        const int nch = 2 + (int)(U(rng) * 7) % 7;
        float lo[8][3], hi[8][3];
        bool finite = true;
        for (int i = 0; i < nch; ++i)
            for (int k = 0; k < 3; ++k)
            {
                lo[i][k] = 2 * U(rng) - 1;
                hi[i][k] = lo[i][k] + (U(rng) < 0.2f ? 0.0f : U(rng));
                const float u = trial % 2 ? U(rng) : 1.0f;
                if (u < 0.04f) hi[i][k] = INFINITY;
                else if (u < 0.08f) lo[i][k] = -INFINITY;
                else if (u < 0.10f) lo[i][k] = NAN;
                else if (u < 0.12f) lo[i][k] = hi[i][k] = NAN;
                finite = finite && std::isfinite(lo[i][k]) && std::isfinite(hi[i][k]);
            }
        ++nodes;
        unusual += !finite;
        // the child to open: every lane offers its own
        double best[8];
        int pick[8];
        for (int i = 0; i < 8; ++i)
        {
            best[i] = i < nch ? open_area(lo[i], hi[i]) : -1.0;
            pick[i] = i;
        }
        int widest = 0;
        for (int i = 1; i < 8; ++i)
            if (best[i] > best[widest]) widest = i;
        const double most = best[widest];
        for (int x = 4; x > 0; x >>= 1)
        {
            double b[8];
            int p[8];
            for (int i = 0; i < 8; ++i)
            {
                const bool take = opens_before(best[i ^ x], pick[i ^ x], best[i], pick[i]);
                b[i] = take ? best[i ^ x] : best[i];
                p[i] = take ? pick[i ^ x] : pick[i];
            }
            for (int i = 0; i < 8; ++i)
            {
                best[i] = b[i];
                pick[i] = p[i];
            }
        }
        for (int i = 0; i < 8; ++i)
        {
            if (pick[i] != pick[0] || !(best[i] == best[0])) ++disagree;
            if (finite && (pick[i] != widest || best[i] != most)) ++differ;
        }
        // octant slots
        float nlo[3], nhi[3];
        for (int k = 0; k < 3; ++k)
        {
            nlo[k] = FLT_MAX;
            nhi[k] = -FLT_MAX;
            for (int i = 0; i < nch; ++i)
            {
                nlo[k] = fminf(nlo[k], lo[i][k]);
                nhi[k] = fmaxf(nhi[k], hi[i][k]);
            }
        }
        double off[8][3];
        for (int i = 0; i < nch; ++i)
            for (int k = 0; k < 3; ++k)
                off[i][k] = 0.5 * ((double)lo[i][k] + hi[i][k]) - 0.5 * ((double)nlo[k] + nhi[k]);
        unsigned taken[8] = {};
        int slot[8], want_slot[8];
        unsigned want_taken = 0u;
        for (int i = 0; i < 8; ++i) slot[i] = want_slot[i] = -1;
        for (int round = 0; round < nch; ++round)
        {
            double bc[8];
            int bs[8], who[8];
            for (int i = 0; i < 8; ++i)
            {
                bc[i] = -DBL_MAX;
                bs[i] = 8;
                if (i < nch && slot[i] < 0)
                    for (int s = 0; s < 8; ++s)
                    {
                        if ((taken[i] >> s) & 1u) continue;
                        const double c = slot_cost(off[i], s);
                        if (bs[i] == 8 || c > bc[i])
                        {
                            bc[i] = c;
                            bs[i] = s;
                        }
                    }
                who[i] = bs[i] < 8 ? i : 8 + i;
            }
            for (int x = 4; x > 0; x >>= 1)
            {
                double c[8];
                int w[8], s[8];
                for (int i = 0; i < 8; ++i)
                {
                    const bool take = placed_before(bc[i ^ x], who[i ^ x], bc[i], who[i]);
                    c[i] = take ? bc[i ^ x] : bc[i];
                    w[i] = take ? who[i ^ x] : who[i];
                    s[i] = take ? bs[i ^ x] : bs[i];
                }
                for (int i = 0; i < 8; ++i)
                {
                    bc[i] = c[i];
                    who[i] = w[i];
                    bs[i] = s[i];
                }
            }
            for (int i = 0; i < 8; ++i)
            {
                if (who[i] != who[0] || bs[i] != bs[0]) ++disagree;
                taken[i] |= 1u << bs[i];
                if (i == who[i]) slot[i] = bs[i];
            }
            // the serial choice: the best (child, slot) left, the earliest of equal ones
            int wi = -1, ws = -1;
            double wc = 0.0;
            for (int i = 0; i < nch; ++i)
                for (int s = 0; s < 8 && want_slot[i] < 0; ++s)
                {
                    if ((want_taken >> s) & 1u) continue;
                    double c = 0.0;
                    for (int k = 0; k < 3; ++k) c += ((s >> k) & 1) ? off[i][k] : -off[i][k];
                    if (wi < 0 || c > wc)
                    {
                        wc = c;
                        wi = i;
                        ws = s;
                    }
                }
            want_slot[wi] = ws;
            want_taken |= 1u << ws;
        }
        unsigned used = 0u;
        for (int i = 0; i < nch; ++i)
        {
            if (slot[i] < 0 || slot[i] > 7 || ((used >> slot[i]) & 1u)) ++lost;
            else used |= 1u << slot[i];
            if (finite && slot[i] != want_slot[i]) ++differ;
        }
    }
    std::printf("%lld %lld %lld %lld %lld\n", nodes, unusual, disagree, lost, differ);
    return 0;
}
"""


def test_lanes_agree(tmp_path):
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    if not nvcc.exists():
        nvcc = shutil.which("nvcc")
        if nvcc is None:
            pytest.skip("nvcc not found")
    src = tmp_path / "lanes.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "lanes"
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-fmad=false", "-Xcompiler", "-ffp-contract=off", "-I", str(CSRC),
                    str(src), "-o", str(exe)], check=True)
    nodes, unusual, disagree, lost, differ = map(int, subprocess.run([str(exe)], check=True, capture_output=True,
                                                                    text=True).stdout.split())
    assert nodes == 200_000 and unusual > 80_000
    assert disagree == 0, f"lanes ended with different winners {disagree} times"
    assert lost == 0, f"{lost} children without a slot of their own"
    assert differ == 0
