"""The two renders of large chunks (tiles, csrc/disc_tile.cu, and segments,
csrc/disc_seg.cu) each by itself, chosen with the tuning's large_render,
against the FP64 oracle.

Bounds: those of the compensated form in test_gpu_configs.py (its check()).
The segmented render adds FP32 deposits into an FP32 plane, up to about 512 a
pixel and segment, each addition rounding by 1.7e-8 rms of the running total: 2.2e-7 of a
pixel's total at most and, as the pixels' errors have either sign, 2e-10 of
the flux for the 786,432 pixels of the smaller map.
"""
import functools

import numpy as np
import pytest

import annmap
from annmap import synth
from test_gpu_configs import check, oracle_map

pytestmark = pytest.mark.gpu

COMP, PLAIN = annmap.COMP_F32, annmap.PLAIN_F64
ANY, TILES, SEGMENTS = 1, 2, 3


@functools.lru_cache(maxsize=None)
def oracle_case(case):
    if case == "halo20k_ns256":
        # 1.2e9 deposits over many octaves of the deposit scale, more than 512
        # a pixel in the largest: a plan of many segments, octaves split among several
        P, nside = synth.nfw_halo(20000, seed=4711, n_sub=6), 256
    else:
        P, nside = synth.workload("nfw16m_sub100_ns2048")
        P = P.subset(slice(0, 1 << 15))
    return P, nside, oracle_map(P, nside)


@pytest.mark.parametrize("case", ["halo20k_ns256", "nfw16m_prefix"])
@pytest.mark.parametrize("large,threads", [(TILES, 256), (SEGMENTS, 128), (SEGMENTS, 256)])
def test_render_by_itself(case, large, threads):
    P, nside, (o, ref, ost, tot) = oracle_case(case)
    with annmap.Renderer(0) as r:
        r.set_tuning(seg_min_deposits_log2=1, block_threads=threads, large_render=large)
        r.set_params(annmap.Parameters.for_synthetic(P, nside))
        got = r.render(P.as_dict(), nside, COMP)
        st = r.stats()
    check(got, ref, tot, o.dOmega, COMP, f"{case} render {large} {threads} threads", nside)
    assert st["deposits"] == ost["deposits"]
    assert st["pass2_ms"] > 0.0
    assert (st["launches"] > 100) == (large == SEGMENTS)   # the segments' slots


def test_tiles_without_room_for_the_pairs():
    """A chunk with more pairs than the tiles' list holds and no segments to
    take it: the per-disc kernels render it.  Every disc but the first has a
    flux of 0, so the map is that of one disc."""
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
        r.set_tuning(large_render=TILES)
        got = r.render(parts, nside, COMP)
        st = r.stats()
        one = r.render({k: v[:1] for k, v in parts.items()}, nside, PLAIN)
    assert st["pass2_ms"] == 0.0
    assert np.array_equal(got != 0, one != 0)
    m = one > 0
    assert (np.abs(got[m] - one[m]) / one[m]).max() <= 1e-5
    assert abs(got.sum() - one.sum()) <= 6e-8 * one.sum()
