"""The exact scatter kernel's split into CTAs of 4, 2 or 1 voxel columns: every split
gives the same bits.  The sizes cross each line of the dispatch (rows x bricks), with a
ragged last detector tile, brick and y run; the values themselves are checked against the
reference's and the oracle's in test_scatter_gpu.py."""
import numpy as np
import pytest

import sysmat_b200
from sysmat_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def full():
    ctx = sysmat_b200.Context(0)
    geo = sysmat_b200.Geometry(ctx, configs.scatter_geometry((19, 37, 9)))   # 3 x 2 x 9 bricks
    rng = np.random.default_rng(4)
    pe = np.exp(rng.normal(-12.0, 3.0, (geo.n_crystals, 19 * 37 * 9))).astype(np.float32)
    pe[rng.random(pe.shape) < 0.3] = 0.0
    pe[rng.random(geo.n_crystals) < 0.1] = 0.0
    yield geo, pe, {part: geo.scatter(pe=pe, parts=part) for part in ("crystal", "collimator")}
    geo.close()
    ctx.close()


@pytest.mark.parametrize("part", ["crystal", "collimator"])
@pytest.mark.parametrize("rows", [(700, 1403), (33, 350), (1024, 1200), (2047, 2048)])   # 4, 4, 2 and 1 columns
def test_every_split_gives_the_same_bits(full, part, rows):
    geo, pe, matrix = full
    assert np.isfinite(matrix[part]).all() and (matrix[part] > 0).any()
    assert np.array_equal(geo.scatter(pe=pe, parts=part, rows=rows), matrix[part][rows[0]:rows[1]])
