"""The compensated adjoint on either side of the set size from which its blocks
have 128 threads instead of 256 (csrc/disc_comp.cu): a particle's gradient
does not depend on the others, so the shared particles' gradients are equal but for
the sums' order.  Bounds: each shape's own distance from the exact gradient as
test_gpu_disc_paths.py derives it (1.1e-5 of dL/dm, 2e-5 + 5e-7 / R of the
position's, R a pixel or more: 0.03), twice.
"""
import numpy as np
import pytest

import annmap
from annmap import synth

pytestmark = pytest.mark.gpu


def test_both_block_shapes():
    nside, edge = 32, 1 << 18
    P = synth.nfw_halo(edge + 1, seed=77, n_sub=3)
    parts = P.as_dict()
    npix = 12 * nside * nside
    G = 1.0 + 0.5 * np.linspace(-1.0, 1.0, npix)   # smooth over the sky: pixels run from pole to pole
    with annmap.Renderer(0) as r:
        r.set_params(annmap.Parameters.for_synthetic(P, nside))
        narrow, _ = r.adjoint(parts, nside, G, precision=annmap.COMP_F32)
        wide, _ = r.adjoint({k: v[:edge] for k, v in parts.items()}, nside, G, precision=annmap.COMP_F32)
    narrow = narrow[:, :edge]
    assert np.linalg.norm(narrow[3] - wide[3]) <= 2.2e-5 * np.linalg.norm(wide[3])
    assert np.linalg.norm(narrow[:3] - wide[:3]) <= 7.4e-5 * np.linalg.norm(wide[:3])
