"""The per-disc kernels at the sizes where their dispatch changes: the warp
kernel's lanes per ring, the key scan's class boundary, and the plain form's
kept weights and azimuth tables, each as the compensated against the plain
form on single discs.

Tolerances.  A compensated weight's exponent of 2, -K theta^2 in [-8.7, 0],
comes from relative roundings of at most 2^-24 each: K 1, A = hav(theta_r -
theta0) 7, B = sin sin 3, x^2 (x from its offset, step and sum) 7, h 1, the
asin^2 series 4, the product 1: 24 of 6e-8, times 8.7 ln 2, less than 9e-6 of
the weight; ex2 adds 1.2e-7 and the deposit's own rounding 6e-8: 1e-5 per
pixel.  The normalisation is FP32 two-floats and the deposits' roundings have
either sign: 6e-8 of the flux at most.
"""
import math

import numpy as np
import pytest

import annmap
import oracle as O

pytestmark = pytest.mark.gpu

COMP, PLAIN = annmap.COMP_F32, annmap.PLAIN_F64


def disc(theta, phi, radius):
    p = [math.sin(theta) * math.cos(phi), math.sin(theta) * math.sin(phi), math.cos(theta)]
    one = {k: np.array([v], np.float32) for k, v in zip("xyz", p)}
    one.update(m=np.ones(1, np.float32), rho=np.ones(1, np.float32), h=np.full(1, radius / 2, np.float32))
    return one


def compare(r, nside, parts):
    got = r.render(parts, nside, COMP)
    st = r.stats()
    ref = r.render(parts, nside, PLAIN)
    sp = r.stats()
    assert np.array_equal(got != 0, ref != 0)
    assert st["deposits"] == sp["deposits"] and st["n_disc_block"] == sp["n_disc_block"]
    m = ref > 0
    assert (np.abs(got[m] - ref[m]) / ref[m]).max() <= 1e-5
    assert abs(got.sum() - ref.sum()) <= 6e-8 * ref.sum()
    return st


@pytest.fixture(scope="module")
def rend():
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        yield r


# mean rings of about 1 to 80 pixels (steps of 8, 16, 32 and 64), more than
# the 64 rings staged at a time, at the seam and over a pole
@pytest.mark.parametrize("pixels", [1.5, 4, 9, 13, 18, 26, 40, 54, 100])
@pytest.mark.parametrize("theta,phi", [(1.3, 3.14159), (0.01, 1.0)])
def test_warp_class(rend, pixels, theta, phi):
    nside = 256
    rend.set_tuning(warp_max_pixels=1 << 20, seg_min_deposits_log2=62)
    st = compare(rend, nside, disc(theta, phi, 0.5 * pixels * math.pi / (2 * nside)))
    assert st["n_disc_block"] == 0


# 1000 discs on either side of a class boundary
@pytest.mark.parametrize("edge", [1, 16, 300, 1 << 20])
def test_class_boundary(rend, edge):
    rng = np.random.default_rng(edge)
    parts = {k: np.concatenate([disc(math.acos(u), p, r)[k] for u, p, r in zip(
        rng.uniform(-1, 1, 1000), rng.uniform(0, 6.28, 1000), np.exp(rng.uniform(-5, -1, 1000)))])
        for k in ("x", "y", "z", "m", "rho", "h")}
    rend.set_tuning(warp_max_pixels=edge, seg_min_deposits_log2=62)
    st = compare(rend, 64, parts)
    assert 0 < st["n_disc"] <= 1000


# a disc within the scratch, one beyond it; Nside without a cap table, over the
# pole and in the belt; both kernels
@pytest.mark.parametrize("nside,theta,radius", [(64, 1.0, 0.3), (512, 1.2, 1.0), (1024, 0.3, 0.6),
                                                (1500, 0.01, 0.02), (1500, 1.5, 0.05)])
@pytest.mark.parametrize("edge", [64, 1 << 28])
def test_plain_form(rend, nside, theta, radius, edge):
    rend.set_tuning(warp_max_pixels=edge, seg_min_deposits_log2=62)
    parts = disc(theta, 2.0, radius)
    compare(rend, nside, parts)
    # the FP64 adjoint keeps its own weights: dL/dm m = L for L = sum G map
    G = np.random.default_rng(1).uniform(0.5, 1.5, 12 * nside * nside)
    grad, _ = rend.adjoint(parts, nside, G, precision=PLAIN)
    L = float(G @ rend.render(parts, nside, PLAIN))
    assert abs(grad[3, 0] - L) <= 1e-9 * L


@pytest.fixture(scope="module")
def vectors():
    h = O.Healpix(128)
    return np.array([h.pix2vec(p) for p in range(h.npix)])


# The compensated adjoint of one disc in each pair of polynomial lengths that a
# disc can have, by either kernel.  L = sum G map is linear in m, and its error
# that of the weights (1e-5 of each, above) times G's range over G (at most 1)
# and G's rounding: 1.1e-5.  G rises linearly along a tangent t, so the terms
# (G - Gm) w e of the position's gradient are aligned: the weights' 1e-5 grows
# by E|e_t||e| / E e_t^2 = 1.3 to 2e-5 with the tangent's own roundings, and G
# and Gm, rounded to 6e-8 of 1.5, against 0.2 R: 5e-7 / R.
@pytest.mark.parametrize("theta,radius", [(1.5, 0.03), (1.5, 0.1), (1.5, 0.2), (1.5, 0.5), (0.05, 0.1),
                                          (1.2, 2.5)])
@pytest.mark.parametrize("edge", [64, 1 << 28])
def test_adjoint_tiers(rend, vectors, theta, radius, edge):
    nside, phi = 128, 2.0
    rend.set_tuning(warp_max_pixels=edge, seg_min_deposits_log2=62)
    parts = disc(theta, phi, radius)
    t = np.array([math.cos(theta) * math.cos(phi), math.cos(theta) * math.sin(phi), -math.sin(theta)])
    G = 1.0 + 0.5 * (vectors @ t)
    got, _ = rend.adjoint(parts, nside, G, precision=COMP)
    ref, _ = rend.adjoint(parts, nside, G, precision=PLAIN)
    assert abs(got[3, 0] - ref[3, 0]) <= 1.1e-5 * abs(ref[3, 0])
    assert np.linalg.norm(got[:3] - ref[:3]) <= (2e-5 + 5e-7 / radius) * np.linalg.norm(ref[:3])


# Host maps on either side of the size from which their pages are touched ahead
# of the copy (4 MB: Nside 209), fresh and at an odd offset in a larger buffer
# whose neighbours stay as they are; the sums are FP64 in an order of their own.
@pytest.mark.parametrize("nside", [64, 209, 300])
def test_host_map(rend, nside):
    torch = pytest.importorskip("torch")
    rend.set_tuning(seg_min_deposits_log2=62)
    parts = disc(1.0, 2.0, 0.7)
    npix = 12 * nside * nside
    dev = torch.zeros(npix, dtype=torch.float64, device="cuda")
    rend.render({k: torch.from_numpy(v).cuda() for k, v in parts.items()}, nside, PLAIN, out=dev)
    buf = np.full(npix + 2, -7.0)
    rend.render(parts, nside, PLAIN, out=buf[1:-1])
    assert buf[0] == -7.0 and buf[-1] == -7.0
    for got in (buf[1:-1], rend.render(parts, nside, PLAIN)):
        np.testing.assert_allclose(got, dev.cpu().numpy(), rtol=1e-12, atol=0)
