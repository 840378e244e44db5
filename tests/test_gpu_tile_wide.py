"""The tiled render's tallest discs (more than 96 strips of 32 rings), whose
strips of the pair list are dealt to many warps: next to shorter discs, over the
poles, over the whole sky, and at azimuths where a full ring's first pixel
changes, against the plain FP64 form; and the time of one against the segmented
render's, which has no pair list.

Tolerances: those of compare() in test_gpu_tiles.py; the flux of giants is off
by 1e-12 and that of 300 discs by 5e-9 / sqrt(300).  The time: both renders
evaluate every pixel of the disc twice, and tiles may take twice as long (with
the 130,000 pairs of the disc on 8 lanes they took 2.2 times as long).
"""
import math

import numpy as np
import pytest

import annmap
from test_gpu_tiles import compare

pytestmark = pytest.mark.gpu


def discs(theta, phi, radius):
    theta, phi = np.asarray(theta, float), np.asarray(phi, float)
    one = np.ones(len(theta), np.float32)
    return dict(x=(np.sin(theta) * np.cos(phi)).astype(np.float32), y=(np.sin(theta) * np.sin(phi)).astype(np.float32),
                z=np.cos(theta).astype(np.float32), m=one, rho=one, h=one * (np.asarray(radius, np.float32) / 2))


@pytest.fixture(scope="module")
def rend():
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        yield r


# Nside 776 has 97 strips: only discs over the whole sky are dealt out
@pytest.mark.parametrize("nside", [775, 776, 1024])
def test_giants(rend, nside):
    # over the whole sky, over a pole, over both, about the equator, and short ones
    theta = [0.3, 1.2, 2.9, 1.57, 0.02, 1.0, 2.0]
    phi = [0.0, math.pi, 2.0 * math.pi - 1e-6, math.pi / 2, 1.0, 4.0, 5.0]
    compare(rend, discs(theta, phi, [3.3, 2.5, 2.0, 1.54, 1.3, 0.4, 0.1]), nside, 1e-9)


def test_long_discs(rend):
    rng = np.random.default_rng(5)
    n = 300   # none with 1/256 of the flux
    compare(rend, discs(np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * math.pi, n), rng.uniform(1.0, 2.1, n)),
            1024, 1e-9)


# phi such that nr (phi / 2 pi - 1 / 2) - shift is an integer, or just beside one
@pytest.mark.parametrize("k", range(8))
@pytest.mark.parametrize("off", [-1e-7, 0.0, 1e-7])
def test_full_rings(rend, k, off):
    nside = 64
    compare(rend, discs([0.4, 2.8], [k * math.pi / 4 + off + 1e-3, (k + 0.5) * 2 * math.pi / (4 * nside) + off],
                        [2.4, 3.2]), nside, 1e-9)


def test_time_of_an_all_sky_disc(rend):
    torch = pytest.importorskip("torch")
    nside = 4096
    out = torch.empty(12 * nside * nside, dtype=torch.float64, device="cuda")
    parts = {k: torch.from_numpy(v).cuda() for k, v in discs([1.0], [2.0], [3.2]).items()}
    t = {}
    for large in (2, 3):
        rend.set_tuning(seg_min_deposits_log2=1, large_render=large)
        ms = []
        for _ in range(7):
            rend.render(parts, nside, annmap.COMP_F32, out=out)
            st = rend.stats()
            ms.append(st["pass1_ms"] + st["pass2_ms"])
        t[large] = sorted(ms)[3]
    rend.set_tuning(seg_min_deposits_log2=28, large_render=1)
    assert 0.0 < t[2] <= 2.0 * t[3], t
