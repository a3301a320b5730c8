"""The hit lists of every form of the photoelectric kernel (few or many rays per entry,
several voxels per group, detectors without and with rotated crystals) against the oracle's,
ray by ray, and the counting form's matrix, which tests one crystal at a time in its own
frame, against the plain forms', bit for bit: the same operations in the same order."""
import numpy as np
import pytest

import oracle_py
import sysmat_b200
from sysmat_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotated", [None, 0, 7])
@pytest.mark.parametrize("sv,sc", [((1, 1, 1), (2, 4, 2)), ((2, 1, 1), (2, 2, 2)), ((2, 2, 1), (1, 4, 1)),
                                   ((2, 2, 2), (2, 4, 2)), ((3, 1, 1), (1, 5, 3)), ((1, 1, 1), (5, 4, 4))])
@pytest.mark.parametrize("layers", [2, 5])
def test_hit_lists_of_all_forms(layers, sv, sc, rotated):
    p = configs.tiny(seed=6, layers=layers)
    p.sv, p.sc = sv, sc
    if rotated is not None:
        p.detector[1 + 12 * rotated + 11] = 0.2
    ctx = sysmat_b200.Context(0)
    g = sysmat_b200.Geometry(ctx, p)
    rng = np.random.default_rng(1)
    # from the rear layers, whose rays cross the most crystals; voxels side by side share a group
    n = p.n_crystals
    rows = np.sort(rng.integers(n // 2, n, 6)).repeat(4)
    vox = (rng.integers(0, p.n_voxels - 4, 6)[:, None] + np.arange(4)).ravel()
    rec = g.record_hits(rows, vox)
    crystals = 0
    for i in range(len(rows)):
        mine = sysmat_b200.parse_records(rec[i])
        ref = oracle_py.parse_hits(oracle_py.oracle_pe_hits(p, int(rows[i]), int(vox[i])))
        assert mine == ref, (rows[i], vox[i])
        crystals += sum(len(c) for _, _, c in ref.values())
    assert crystals > 0
    A = g.pe()
    ctx.set_counters(True)
    assert np.array_equal(g.pe(), A)
    g.close()
    ctx.close()
