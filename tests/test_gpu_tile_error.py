"""The tiled render's pixels are no further from the plain FP64 form than the
segmented render's, which deposits w (F + Flo) with a two-float scale and a
full-length polynomial: the 2-norm of the error over some 1e6 pixels, most of it
from the discs' bright centres (known to 0.2 %; 5 % leaves room for the tiles' and the
plane's different sums where discs overlap).  The discs hardly overlap, so that
the errors are those of single deposits; no disc has 1/256 of the flux.
"""
import math

import numpy as np
import pytest

import annmap
from annmap import synth

pytestmark = pytest.mark.gpu

COMP, PLAIN = annmap.COMP_F32, annmap.PLAIN_F64
TILES, SEGMENTS = 2, 3


@pytest.fixture(scope="module")
def rend():
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        yield r


# radii: exponents whose y^4 term is far below rounding
@pytest.mark.parametrize("nside,n,lo,hi", [(512, 600, 0.045, 0.055), (2048, 600, 0.02, 0.05)])
def test_pixel_errors(rend, nside, n, lo, hi):
    rng = np.random.default_rng(5)
    z, phi, radius = rng.uniform(-0.9, 0.9, n), rng.uniform(0, 2 * math.pi, n), rng.uniform(lo, hi, n)
    s = np.sqrt(1.0 - z * z)
    parts = {"x": s * np.cos(phi), "y": s * np.sin(phi), "z": z, "m": rng.uniform(1.0, 1.2, n),
             "rho": rng.uniform(1.0, 1.2, n), "h": radius / 2}
    parts = {k: v.astype(np.float32) for k, v in parts.items()}
    ref = rend.render(parts, nside, PLAIN)
    err = {}
    for large in (TILES, SEGMENTS):
        rend.set_tuning(seg_min_deposits_log2=1, warp_max_pixels=16, large_render=large)
        got = rend.render(parts, nside, COMP)
        assert rend.stats()["pass2_ms"] > 0.0
        err[large] = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    print("error", err)
    assert err[TILES] <= 1.05 * err[SEGMENTS]


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_dense_map(rend, seed):
    """A third of a million particles of a halo of four: thousands of deposits in
    the bright pixels, whose FP32 sums (of at most 128 discs, tile_plan.h) are
    then the error; 10 % for the luck of the brightest few."""
    n, nside = 346889, 742
    P = synth.nfw_halo(n, seed=seed, n_total=1 << 22, near_observer=20)
    with annmap.Renderer(0) as r:
        r.set_params(annmap.Parameters.for_synthetic(P, nside))
        ref = r.render(P.as_dict(), nside, PLAIN)
        err = {}
        for large in (TILES, SEGMENTS):
            r.set_tuning(large_render=large)
            got = r.render(P.as_dict(), nside, COMP)
            assert r.stats()["pass2_ms"] > 0.0
            err[large] = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    print("error", err)
    assert err[TILES] <= 1.1 * err[SEGMENTS]
