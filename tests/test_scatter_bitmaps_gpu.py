"""Bitmap words and pair sums at detector sizes that are no multiple of the 32 bits of a
word: the words equal the oracle's, and scatter from given bitmaps equals scatter that
decides the bits where a crystal is crossed."""
import numpy as np
import pytest

import oracle_py
import sysmat_b200
from sysmat_b200 import configs
from sysmat_b200.params import Params, build_collimator, build_detector, build_image, build_physics, crystal_layer, grid_holes

pytestmark = pytest.mark.gpu


def geometry(nx, nz, layers, tilt):
    rng = np.random.default_rng(nx * nz + layers)
    col = build_collimator([configs._plate(40.0, 4.0, 40.0, 0.0, grid_holes(3, 3, 5.0, 0.6, 4.0, 0.0, jitter=0.6, rng=rng))])
    crystals = [c for l in range(layers) for c in crystal_layer(nx, nz, 2.0, (2.0, 4.0, 2.0), 14.0 + 4.5 * l)]
    for c in crystals:
        c.rotation = float(rng.uniform(-tilt, tilt))
    return Params(col, build_detector(crystals), build_image((6, 5, 4), (2.0, 2.0, 2.0), fov_to_plate0=20.0), build_physics())


@pytest.mark.parametrize("nx,nz,layers,tilt", [(1, 1, 1, 0.0), (3, 1, 1, 0.0), (7, 5, 1, 0.0), (9, 7, 1, 0.2), (6, 11, 2, 0.0)])
def test_words_and_scatter_at_ragged_sizes(nx, nz, layers, tilt):
    p = geometry(nx, nz, layers, tilt)
    ctx = sysmat_b200.Context(0)
    geo = sysmat_b200.Geometry(ctx, p)
    try:
        crystal, collimator = geo.scatter_bitmaps()
        want_c, want_h = oracle_py.oracle_bitmap_crystal(p), oracle_py.oracle_bitmap_collimator(p)
        assert np.array_equal(crystal, want_c) and np.array_equal(collimator, want_h)
        pe = geo.pe(opts=sysmat_b200.PeOptions.make((1, 1, 1), (2, 4, 2)))
        for sp in ((1, 1, 1), (2, 3, 1)):
            here = geo.scatter(pe=pe, sp=sp)
            assert np.isfinite(here).all()
            assert np.array_equal(here, geo.scatter(pe=pe, sp=sp, bitmaps=(crystal, collimator)))
    finally:
        geo.close()
        ctx.close()
