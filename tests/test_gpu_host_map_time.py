"""Fresh host maps against the plain way to one: the map rendered on the device
and copied into a fresh array.  Preparing the array's pages ahead of the copy
must not cost more than the copy's own page faults did: a pass that read each
page before it wrote to it took 40 ms at this size, nine times the plain way.

The bound is twice the plain way's median (which renders the same map and makes
the same pages) and a millisecond for the call itself.
"""
import time

import numpy as np
import pytest

import annmap

pytestmark = pytest.mark.gpu


def test_fresh_host_map_takes_no_longer_than_a_copy():
    torch = pytest.importorskip("torch")
    nside = 1024
    npix = 12 * nside * nside
    parts = {k: torch.full((1,), v, device="cuda") for k, v in
             zip(("x", "y", "z", "m", "rho", "h"), (0.6, 0.0, 0.8, 1.0, 1.0, 0.05))}
    with annmap.Renderer(0) as r:
        r.set_frame(np.eye(3), (0.0, 0.0, 0.0))
        r.set_units(1.0)
        dev = torch.empty(npix, dtype=torch.float64, device="cuda")

        def plain():
            r.render(parts, nside, annmap.COMP_F32, out=dev)
            out = np.zeros(npix)
            torch.from_numpy(out).copy_(dev)
            return out

        def fresh():
            return r.render(parts, nside, annmap.COMP_F32)

        def median(call):
            t = []
            for _ in range(9):
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                out = call()
                t.append(time.perf_counter() - t0)
            return sorted(t)[4], out

        median(plain)
        tp, want = median(plain)
        tf, got = median(fresh)
    assert np.array_equal(got, want)
    assert tf <= 2 * tp + 1e-3, (tf, tp)
