"""The bilateral filter's quick pair tests and its two tile heights, against a
float64 restatement of the filter (the reference's formulas, radius 7, clamped
neighbours): image sizes at tile edges and on both sides of the switch between
tile heights, few and many samples, different sample counts in one image, and
noise-free regions.

Tolerance: a float filter over 225 taps differs from float64 by at most about
225 roundings of the colour and weight sums (225 * 2^-23 = 2.7e-5 relative) plus the
tested difference of nearly equal thetas; a pair whose t statistic lies within
that of its threshold may fall on the other side, which moves a pixel by up to
one tap's weight.  So 99 % of the values agree within 1e-4 and the image within
1e-3 (2-norm)."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, configs
from aperturerendererv3_gb300._lib import DENOISE_GBUF_DTYPE, DENOISE_STAT_DTYPE

pytestmark = pytest.mark.gpu

stats = pytest.importorskip("scipy.stats")


def _records(w, h, spp, seed, mixed, flat):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    reg = ((4 * x) // max(1, w) + (3 * y) // max(1, h)) % 5
    g, s = np.zeros((h, w), DENOISE_GBUF_DTYPE), np.zeros((h, w), DENOISE_STAT_DTYPE)
    n = rng.normal(size=(5, 3))[reg] + rng.normal(0.0, 0.02, (h, w, 3))
    half = np.zeros((h, w, 14))
    half[..., 0:3] = rng.uniform(0.1, 0.9, (5, 3))[reg]
    half[..., 3:6] = n / np.linalg.norm(n, axis=-1, keepdims=True)
    half[..., 6], half[..., 7] = rng.choice([0.0, 1.0], 5)[reg], rng.uniform(0.05, 1.0, 5)[reg]
    half[..., 8], half[..., 11] = 0.25 * reg / 4.0, 1.0 - 0.25 * reg / 4.0
    g["h"] = half.astype(np.float16).view(np.uint16)
    g["depth"] = 1.0 + 0.3 * x / w + rng.normal(0.0, 1e-3, (h, w))
    count = rng.integers(max(2, spp // 2), 2 * spp + 1, (h, w)) if mixed else np.full((h, w), spp)
    g["valid"] = g["frames"] = s["num"] = count
    level = rng.uniform(0.05, 2.0, (5, 1))[reg] * np.array([0.9, 1.0, 1.1])
    sd = 0.3 * level
    c = count[..., None]
    s["mean"] = 2.0 * (np.sqrt(level) - 1.0) + rng.normal(size=(h, w, 3)) * sd / np.sqrt(c)
    s["m2n"] = sd ** 2 * rng.gamma(np.maximum(1.0, (c - 1) / 2.0), 2.0 / np.maximum(1, c - 1), (h, w, 3)) + 1e-6
    s["m3n"] = sd ** 3 * rng.normal(0.0, 0.3, (h, w, 3))
    if flat:
        s["m2n"][reg == 0] = 0.0  # no noise: theta is not a number there
        s["m3n"][reg == 0] = 0.0
    xyz = np.maximum(1.0 + s["mean"].astype(np.float64) / 2.0, 0.0) ** 2
    return g, s, xyz


def _filter64(g, s, xyz):
    half = g["h"].view(np.float16).astype(np.float64)
    alb, nrm, mr, model = half[..., 0:3], half[..., 3:6], half[..., 6:8], half[..., 8:13]
    nrm = nrm / np.linalg.norm(nrm, axis=-1, keepdims=True)
    dep, num = g["depth"].astype(np.float64), s["num"].astype(np.float64)[..., None]
    with np.errstate(all="ignore"):
        var = s["m2n"].astype(np.float64) * num / np.maximum(num - 1, 1)
        vth = var / num
        theta = s["mean"].astype(np.float64) + s["m3n"].astype(np.float64) / 6.0 / var
        lo = vth ** 2 / np.maximum(num - 1, 1)
        tq = stats.t.ppf(1.0 - 0.0025, np.arange(1, 1025))
        col = np.log1p(xyz)
        h, w = dep.shape
        acc, ws = col * 1e-6, np.full((h, w), 1e-6)
        for dj in range(-7, 8):
            for di in range(-7, 8):
                ix = np.ix_(np.clip(np.arange(h) + dj, 0, h - 1), np.clip(np.arange(w) + di, 0, w - 1))
                t2 = (theta - theta[ix]) ** 2
                stat = np.sqrt(0.5 / (1.0 - (t2 + vth[ix]) / np.maximum(t2 + vth + vth[ix], 1e-6)) - 1.0)
                nu = (vth + vth[ix]) ** 2 / (lo + lo[ix])
                q = tq[np.clip(np.nan_to_num(np.floor(nu)).astype(np.int64), 1, 1024) - 1]
                keep = (stat < q).all(-1)
                b = dep[ix]
                term = 0.5 * ((alb - alb[ix]) ** 2).sum(-1) + 2.0 * (1.0 - (nrm * nrm[ix]).sum(-1)) ** 2
                term = term + 8.0 * ((dep - b) / np.maximum(np.maximum(dep, b), 1e-6)) ** 2
                term = term + 2.0 * ((mr - mr[ix]) ** 2).sum(-1) + 50.0 * (0.5 * np.abs(model - model[ix]).sum(-1)) ** 2
                wt = np.where(keep, np.exp(-term - 0.125 * (di * di + dj * dj)), 0.0)
                acc, ws = acc + col[ix] * wt[..., None], ws + wt
    return np.maximum(np.expm1(acc / ws[..., None]), 0.0)


@pytest.mark.parametrize("size,spp,mixed,flat", [
    ((1, 1), 8, False, False), ((31, 33), 2, False, False), ((33, 8), 3, True, False), ((70, 9), 64, False, True),
    ((200, 150), 8, False, False), ((97, 131), 1500, True, True), ((640, 480), 8, False, False),
    ((513, 330), 33, True, True)])
def test_filter_against_float64(cuda_device, size, spp, mixed, flat):
    w, h = size
    g, s, xyz = _records(w, h, spp, 3 + w, mixed, flat)
    r = SceneRenderer(configs.cornell_triangles())
    r.set_denoise_records(g, s)
    out = r.denoise(xyz)
    want = _filter64(g, s, xyz)
    err = np.abs(out - want) / np.maximum(np.abs(want), 1e-3)
    assert np.mean(err <= 1e-4) >= 0.99
    assert np.linalg.norm(out - want) <= 1e-3 * np.linalg.norm(want)
