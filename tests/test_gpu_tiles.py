"""The tiled render (csrc/disc_tile.cu) at the edges of its tiles and of its
dispatch, against the plain FP64 form on the same particles: the same set of
non-zero pixels, the same deposit count, every pixel and the total flux.

Tolerances.  A weight's exponent of 2, in [-8.7, 0], carries some 24 relative
roundings of at most 2^-24 (test_gpu_disc_paths.py), 9e-6 of the weight; a
pixel adds FP32 sums of at most 512 deposits, whose roundings have either sign:
1e-5 per pixel.  The total flux is that of the per-particle normalisation, 1e-9 (the
bound of the other tests); a single disc's normalisation comes from ring sums
rounded to FP32 (6e-8 each, of either sign, over ten rings and more): 6e-8.
"""
import math

import numpy as np
import pytest

import annmap
from annmap import synth

pytestmark = pytest.mark.gpu

COMP, PLAIN = annmap.COMP_F32, annmap.PLAIN_F64


def compare(r, parts, nside, flux_tol):
    r.set_tuning(seg_min_deposits_log2=1, warp_max_pixels=16)
    got = r.render(parts, nside, COMP)
    st = r.stats()
    assert st["pass2_ms"] > 0.0
    ref = r.render(parts, nside, PLAIN)
    sp = r.stats()
    assert np.array_equal(got != 0, ref != 0)
    assert st["deposits"] == sp["deposits"]
    m = ref > 1e-6 * ref.max()
    assert (np.abs(got[m] - ref[m]) / ref[m]).max() <= 1e-5
    assert abs(got.sum() - ref.sum()) <= flux_tol * ref.sum()


# Nside whose rings and in-ring pixels are no multiples of the tile's, few tiles
# for the whole map, several columns, and rings fine enough for the
# interpolated general discs
@pytest.mark.parametrize("nside", [24, 100, 256, 317])
def test_halo(nside):
    P = synth.nfw_halo(3000, seed=900 + nside, n_sub=3, n_total=3000 * max(1, nside // 24), near_observer=5)
    with annmap.Renderer(0) as r:
        r.set_params(annmap.Parameters.for_synthetic(P, nside))
        compare(r, P.as_dict(), nside, 1e-9)


def disc(theta, phi, radius):
    p = [math.sin(theta) * math.cos(phi), math.sin(theta) * math.sin(phi), math.cos(theta)]
    one = {k: np.array([v], np.float32) for k, v in zip("xyz", p)}
    one.update(m=np.ones(1, np.float32), rho=np.ones(1, np.float32), h=np.full(1, radius / 2, np.float32))
    return one


# single discs: at the seam of the ring index, over and beside the poles, at
# the border of cap and belt, across a strip of tiles, at the largest
# polynomial radius, beyond it, beyond 90 degrees, the whole sky
@pytest.mark.parametrize("nside", [64, 512])
@pytest.mark.parametrize("theta,phi,radius", [
    (1.4, 3.14159, 0.1), (1.4, 3.1, 0.24), (0.002, 1.0, 0.15), (0.2, 3.14, 0.15), (3.0, 2.0, 0.3),
    (0.84, 0.0, 0.12), (2.3, 3.2, 0.27), (1.57, 1.0, 0.31), (1.0, 3.14, 0.7), (0.5, 2.0, 1.3),
    (1.2, 4.0, 2.1), (1.2, 4.0, 2.6), (2.0, 0.5, 3.3)])
def test_single_disc(nside, theta, phi, radius):
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        compare(r, disc(theta, phi, radius), nside, 6e-8)


def test_more_pairs_than_the_list_holds():
    """Discs of most of the sky touch more tiles than the pair list's 96 per
    particle and 2^24: the chunk is rendered in segments.  Every disc but the
    first has a flux of 0 (zero mass), so the map is that of one disc and is
    compared with its tiled render."""
    n, nside = 10000, 1024
    rng = np.random.default_rng(7)
    u = rng.standard_normal((n, 3))
    u = (u / np.linalg.norm(u, axis=1)[:, None]).astype(np.float32)
    parts = {"x": u[:, 0].copy(), "y": u[:, 1].copy(), "z": u[:, 2].copy(), "m": np.zeros(n, np.float32),
             "rho": np.ones(n, np.float32), "h": np.full(n, 1.0, np.float32)}
    parts["m"][0] = 1.0
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        got = r.render(parts, nside, COMP)
        st = r.stats()
        one = r.render({k: v[:1] for k, v in parts.items()}, nside, COMP)
        s1 = r.stats()
    assert np.array_equal(got != 0, one != 0)
    m = one > 0
    assert (np.abs(got[m] - one[m]) / one[m]).max() <= 1e-5
    assert abs(got.sum() - one.sum()) <= 6e-8 * one.sum()
    assert st["launches"] > s1["launches"] + 100   # the segments' slots
