"""The traversal's child-box test (csrc/ar_traverse.cuh) over the whole range of
node scales and direction components, on the host.

The planes of a node are evaluated around an offset of 32768 quantisation steps,
which overflows for large nodes and for small direction components.  A box that a
ray meets in [tmin, tlim] may not be rejected there: the traversal's own step()
runs against random nodes with steps from 2^-126 to 2^120 and rays with ordinary,
zero, negative zero, subnormal and tiny components, and is compared with a slab
test in double precision; sheets of 1 to 1e12 units, some of them squashed to
ribbons, are compared with a test of every triangle in double precision."""
import ctypes as C
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from aperturerendererv3_gb300 import _lib

CSRC = Path(__file__).resolve().parents[1] / "aperturerendererv3_gb300" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "ar_traverse.cuh"
using namespace ar;

struct Box { double lo[3], hi[3]; };

static bool exact_hit(const Box& b, const double o[3], const double d[3], double tmin, double tlim)
{
    double tn = tmin, tf = tlim;
    for (int k = 0; k < 3; ++k)
    {
        if (d[k] == 0.0)
        {
            if (o[k] < b.lo[k] || o[k] > b.hi[k]) return false;
            continue;
        }
        double t0 = (b.lo[k] - o[k]) / d[k], t1 = (b.hi[k] - o[k]) / d[k];
        if (t0 > t1) std::swap(t0, t1);
        tn = std::max(tn, t0);
        tf = std::min(tf, t1);
    }
    return tn <= tf;
}

int main()
{
    std::mt19937 rng(31);
    std::uniform_real_distribution<float> U(0.0f, 1.0f);
    enum { ORDINARY, ZERO, NEGATIVE_ZERO, SUBNORMAL, TINY, THIN, KINDS };
    long long met[KINDS] = {}, missed[KINDS] = {};
    for (int trial = 0; trial < 120000; ++trial)
    {
        const int kind = trial % KINDS;
        const int ax = (int)(U(rng) * 3) % 3;  // the axis of the special component
        ar_wide_node nd;
        std::memset(&nd, 0, sizeof(nd));
        int e[3];
        const int base = kind == THIN ? -30 + (int)(U(rng) * 30) : -126 + (int)(U(rng) * 246);
        for (int k = 0; k < 3; ++k)
        {
            // THIN: a node of any extent that is built along the axis that the ray is perpendicular to
            e[k] = kind == THIN && k == ax ? AR_BVH_MIN_EXP + (int)(U(rng) * (base - AR_BVH_MIN_EXP))
                                           : std::min(119, std::max(-126, base + (int)(U(rng) * 10) - 5));
            nd.e[k] = (uint8_t)(e[k] + 127);
        }
        float p[3];
        for (int k = 0; k < 3; ++k) p[k] = std::ldexp(255.0f, e[k]) * (2 * U(rng) - 1);
        nd.px = p[0];
        nd.py = p[1];
        nd.pz = p[2];
        nd.imask = 0xff;
        nd.child_base = 1;
        Box box[8];
        for (int s = 0; s < 8; ++s)
        {
            nd.meta[s] = (uint8_t)(0x80u | (uint32_t)s);
            for (int k = 0; k < 3; ++k)
            {
                int a = std::min(255, (int)(U(rng) * 256)), b = std::min(255, (int)(U(rng) * 256));
                if (a > b) std::swap(a, b);
                nd.qlo[k][s] = (uint8_t)a;
                nd.qhi[k][s] = (uint8_t)b;
                box[s].lo[k] = (double)p[k] + std::ldexp((double)a, e[k]);
                box[s].hi[k] = (double)p[k] + std::ldexp((double)b, e[k]);
            }
        }
        uint4 nodes[5 * 9];
        std::memset(nodes, 0, sizeof(nodes));
        std::memcpy(nodes, &nd, sizeof(nd));
        TravScene sc;
        std::memset(&sc, 0, sizeof(sc));
        sc.nodes = nodes;
        sc.node_count = 9;
        for (int r = 0; r < 8; ++r)
        {
            const int s_t = (int)(U(rng) * 8) & 7;
            float of[3], df[3];
            double dd[3], len = 0;
            const double far = (r & 1) ? 1000.0 : 3.0;
            for (int k = 0; k < 3; ++k)
            {
                const int pick = (int)(U(rng) * 3);
                const double tgt = pick == 0   ? box[s_t].lo[k]
                                   : pick == 1 ? box[s_t].hi[k]
                                               : box[s_t].lo[k] + U(rng) * (box[s_t].hi[k] - box[s_t].lo[k]);
                of[k] = (float)(tgt + far * std::ldexp(255.0, e[k]) * (2 * U(rng) - 1));
                dd[k] = tgt - (double)of[k];
                len += dd[k] * dd[k];
            }
            len = std::sqrt(len);
            if (len == 0 || !(len < 1e38)) continue;
            for (int k = 0; k < 3; ++k) df[k] = (float)(dd[k] / len);
            if (kind != ORDINARY)
            {
                float v = 0.0f;
                if (kind == NEGATIVE_ZERO) v = -0.0f;
                if (kind == SUBNORMAL) v = std::ldexp(1.0f, -149 + (int)(U(rng) * 23));
                if (kind == TINY) v = std::ldexp(1.0f + U(rng), -126 + (int)(U(rng) * 27));
                df[ax] = kind > NEGATIVE_ZERO && U(rng) < 0.5f ? -v : v;
                of[ax] = (float)(box[s_t].lo[ax] + U(rng) * (box[s_t].hi[ax] - box[s_t].lo[ax]));
            }
            const double o[3] = {of[0], of[1], of[2]}, d[3] = {df[0], df[1], df[2]};
            const float tlim = (r & 2) ? (float)len * 1.01f : INFINITY;
            const float tmin = (r % 3 == 0) ? 0.0f : 1e-4f * (float)len;
            TravState<false> st;
            uint2 stk[AR_TRAV_STACK];
            st.init(sc, v3(of[0], of[1], of[2]), v3(df[0], df[1], df[2]), tmin, tlim, stk);
            st.res.t = tlim;
            st.step(sc, nullptr);
            uint32_t got = 0;
            if (st.node >= 1) got |= 1u << (st.node - 1);
            if (st.sp > 0)
            {
                const uint32_t m = stk[0].y & 0xffu;
                for (int i = 0; i < 8; ++i)
                    if (m & (1u << i)) got |= 1u << (i ^ st.oct);
            }
            for (int s = 0; s < 8; ++s)
            {
                if (!exact_hit(box[s], o, d, (double)tmin, (double)tlim)) continue;
                ++met[kind];
                if (!((got >> s) & 1u)) ++missed[kind];
            }
        }
    }
    for (int k = 0; k < KINDS; ++k) std::printf("%lld %lld\n", met[k], missed[k]);
    return 0;
}
"""
KINDS = ["ordinary", "zero", "negative zero", "subnormal", "tiny", "zero in a thin node"]


def test_no_box_is_rejected_at_any_scale(tmp_path):
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    if not nvcc.exists():
        nvcc = shutil.which("nvcc")
        if nvcc is None:
            pytest.skip("nvcc not found")
    src = tmp_path / "range.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "range"
    subprocess.run([str(nvcc), "-O2", "-std=c++17", "-fmad=false", "-Xcompiler", "-ffp-contract=off", "-I", str(CSRC),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    for kind, line in zip(KINDS, out):
        met, missed = map(int, line.split())
        assert met > 50_000, kind
        assert missed == 0, f"{kind}: {missed} of {met} boxes that the ray meets were rejected"


def sheet(size, n=24, thin=1.0):
    """n x n quads of two triangles each over [-size, size]^2 at y = 0, (2 n^2, 9), x scaled by thin."""
    g = np.linspace(-size, size, n + 1)
    x, z = np.meshgrid(thin * g, g, indexing="ij")
    v = np.stack([x, np.zeros_like(x), z], -1)
    a, b, c, d = v[:-1, :-1], v[1:, :-1], v[1:, 1:], v[:-1, 1:]
    return np.concatenate([np.stack([a, b, c], 2).reshape(-1, 9), np.stack([a, c, d], 2).reshape(-1, 9)]).astype(np.float32)


def sheet_rays(tris, direction, height, n=500):
    """Rays along `direction` (not normalised) at points well inside random triangles."""
    rng = np.random.default_rng(3)
    v = tris.reshape(-1, 3, 3).astype(np.float64)
    w = 0.1 + 0.7 * rng.dirichlet((1.0, 1.0, 1.0), n)
    at = (v[rng.integers(0, len(v), n)] * w[:, :, None]).sum(1)
    d = np.asarray(direction, np.float32)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = at - (height / abs(float(d[1]))) * d.astype(np.float64)
    r[:, 4:7], r[:, 7] = d, np.inf
    return r


def every_triangle(tris, rays):
    """Closest hits (id or -1, t) from a test of every triangle in double precision."""
    v = tris.reshape(-1, 3, 3).astype(np.float64)
    o, d = rays[:, None, 0:3].astype(np.float64), rays[:, None, 4:7].astype(np.float64)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    q = np.cross(d, e2)
    det = (q * e1).sum(-1)
    s = o - v[:, 0]
    with np.errstate(divide="ignore", invalid="ignore"):
        b1 = (q * s).sum(-1) / det
        c = np.cross(s, e1)
        b2 = (c * d).sum(-1) / det
        t = (c * e2).sum(-1) / det
    t = np.where((b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t > 0), t, np.inf)
    i = t.argmin(1)
    best = t[np.arange(len(t)), i]
    return np.where(np.isfinite(best), i, -1).astype(np.int32), best


# size, direction, scale of x
SHEETS = [
    (1.0, (0.0, -1.0, 0.0), 1.0),
    (1.0, (1e-36, -1.0, 0.3), 1.0),
    (1e3, (1e-36, -1.0, 0.3), 1.0),
    (1e3, (-1e-37, -1.0, -1e-40), 1.0),
    (1e7, (1e-30, -1.0, 1e-30), 1.0),
    (8e6, (0.0, -1.0, 0.0), 1.0),
    (9e6, (0.0, -1.0, 0.0), 1.0),
    (9e6, (1e-3, -1.0, 0.0), 1.0),
    (1e8, (0.0, -1.0, 0.0), 1.0),
    (1e8, (-0.0, -1.0, 0.25), 1.0),
    (1e8, (0.5, -1.0, 0.25), 1.0),
    (1e12, (0.0, -1.0, 1e-20), 1.0),
    (1.0, (0.0, -1.0, 0.0), 1e-12),
    (1.0, (0.0, -1.0, 0.0), 1e-25),
    (1.0, (0.0, -1.0, 0.5), 1e-30),
    (1e6, (0.0, -1.0, 0.0), 1e-31),
]


@pytest.mark.parametrize("size,direction,thin", SHEETS)
def test_sheets_answer_as_every_triangle(size, direction, thin):
    tris = sheet(size, thin=thin)
    rays = sheet_rays(tris, direction, 0.5 * size)
    want, want_t = every_triangle(tris, rays)
    assert (want >= 0).all()
    ids, t, visits = np.zeros(len(rays), np.int32), np.zeros(len(rays), np.float32), C.c_int64()
    assert _lib.load().ar_host_trace_closest(tris.ctypes.data, len(tris), rays.ctypes.data, len(rays), ids.ctypes.data,
                                             t.ctypes.data, C.byref(visits)) == 0
    assert np.array_equal(ids, want)
    assert np.allclose(t, want_t, rtol=1e-5)
