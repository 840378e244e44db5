"""Total flux of the tiled render (csrc/disc_tile.cu).  Each disc's weights are
divided by a sum that does not visit the pixels, so the flux of a map shows
that sum's errors; the bound is the 1e-9 of the other tests.
"""
import math

import numpy as np
import pytest

import annmap

pytestmark = pytest.mark.gpu

COMP = annmap.COMP_F32


def discs(z, phi, radius, rng):
    s = np.sqrt(1.0 - z * z)
    n = len(z)
    parts = {"x": s * np.cos(phi), "y": s * np.sin(phi), "z": z, "m": rng.uniform(1.0, 1.3, n),
             "rho": rng.uniform(1.0, 1.3, n), "h": radius / 2}
    return {k: v.astype(np.float32) for k, v in parts.items()}


def flux_error(r, parts, nside):
    r.set_tuning(seg_min_deposits_log2=1, warp_max_pixels=16)
    got = r.render(parts, nside, COMP)
    st = r.stats()
    assert st["pass2_ms"] > 0.0
    return got.sum() * (4.0 * math.pi / len(got)) / st["total_flux"] - 1.0


@pytest.fixture(scope="module")
def rend():
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        yield r


# Discs that hold a pole, so that whole rings lie inside them: small ones, and
# of most of a hemisphere and beyond.  The sums' scatter from disc to disc, some
# 5e-9, is 1e-10 over 3000 discs of similar flux.
@pytest.mark.parametrize("nside,lo,hi", [(512, 0.05, 0.2), (128, 1.4, 2.15), (512, 1.4, 2.15)])
def test_full_rings(rend, nside, lo, hi):
    rng = np.random.default_rng(100)
    n = 3000
    z = np.cos(rng.uniform(0.002, 0.9 * lo, n)) * rng.choice([-1.0, 1.0], n)
    radius = np.exp(rng.uniform(math.log(lo), math.log(hi), n))
    assert abs(flux_error(rend, discs(z, rng.uniform(0, 6.28, n), radius, rng), nside)) <= 1e-9


# A disc that is the whole map's flux is summed over its pixels and deposited in
# two-floats: 2^-46 for each of the sums, the quotient and the deposits, which
# is 1e-13, and FP64 sums of up to 3e6 pixels: 1e-11 leaves ten times that.
@pytest.mark.parametrize("nside", [64, 512])
@pytest.mark.parametrize("theta,phi,radius", [
    (1.4, 3.14159, 0.1), (0.002, 1.0, 0.15), (0.84, 0.0, 0.12), (1.57, 1.0, 0.31), (1.0, 3.14, 0.7),
    (0.5, 2.0, 1.3), (1.2, 4.0, 2.1), (1.2, 4.0, 2.6), (2.0, 0.5, 3.3)])
def test_one_disc(rend, nside, theta, phi, radius):
    parts = discs(np.array([math.cos(theta)]), np.array([phi]), np.array([radius]), np.random.default_rng(1))
    assert abs(flux_error(rend, parts, nside)) <= 1e-11


# The discs of test_gpu_tiles.py's test_single_disc 400 times over, so that none
# has 1/256 of the flux and they take the polynomial and general paths, the
# longer general ones (beyond 256 rings) summed in parts: against one disc of the
# plain form, the same pixels, deposits and bounds.
@pytest.mark.parametrize("nside", [64, 512])
@pytest.mark.parametrize("theta,phi,radius", [
    (1.4, 3.14159, 0.1), (1.4, 3.1, 0.24), (0.002, 1.0, 0.15), (0.2, 3.14, 0.15), (3.0, 2.0, 0.3),
    (0.84, 0.0, 0.12), (2.3, 3.2, 0.27), (1.57, 1.0, 0.31), (1.0, 3.14, 0.7), (0.5, 2.0, 1.3),
    (1.2, 4.0, 2.1), (1.2, 4.0, 2.6), (2.0, 0.5, 3.3)])
def test_copies_of_a_disc(rend, nside, theta, phi, radius):
    n = 400
    one = discs(np.array([math.cos(theta)]), np.array([phi]), np.array([radius]), np.random.default_rng(1))
    parts = {k: np.repeat(v, n) for k, v in one.items()}
    assert abs(flux_error(rend, parts, nside)) <= 6e-8
    got = rend.render(parts, nside, COMP)
    st = rend.stats()
    ref = n * rend.render(one, nside, annmap.PLAIN_F64)
    assert st["deposits"] == n * rend.stats()["deposits"]
    assert np.array_equal(got != 0, ref != 0)
    at = ref > 0
    assert (np.abs(got[at] - ref[at]) / ref[at]).max() <= 1e-5
