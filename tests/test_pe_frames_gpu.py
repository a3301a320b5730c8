"""The photoelectric kernel's forms for detectors without and with rotated crystals, for
entries of few rays (several voxels per group) and of many (crystals tested two at a time:
layers give none, odd and even numbers of candidates).  Against the oracle with the
reference's single-precision decisions and double magnitudes: no decision differs, so the
error is that of single-precision arithmetic, 1e-4 as for the kernel's other tests."""
import numpy as np
import pytest
import torch

import oracle_py
import sysmat_b200
from helpers import rel_err
from sysmat_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rotated", [None, 0, -1])
@pytest.mark.parametrize("sv,sc", [((1, 1, 1), (2, 4, 2)), ((2, 2, 2), (2, 4, 2))])
@pytest.mark.parametrize("layers", [1, 2, 4])
def test_frames_and_candidate_counts(layers, sv, sc, rotated):
    p = configs.tiny(seed=6, layers=layers)
    p.sv, p.sc = sv, sc
    if rotated is not None:   # one crystal's frame, the first or the last
        p.detector[1 + 12 * (rotated % p.n_crystals) + 11] = 0.2
    ctx = sysmat_b200.Context(0)
    g = sysmat_b200.Geometry(ctx, p)
    A = g.pe()
    rng = np.random.default_rng(3)
    rows, vox = rng.integers(0, p.n_crystals, 120), rng.integers(0, p.n_voxels, 120)
    rows[:12] = rotated % p.n_crystals if rotated is not None else 0
    err = rel_err(A[rows, vox], oracle_py.oracle_pe_entries(p, rows, vox, "dual"))
    assert err.size > 0 and err.max() <= 1e-4
    ctx.set_counters(True)    # the counting form: the same rays
    assert np.allclose(g.pe(), A, rtol=1e-4, atol=1e-30)
    assert ctx.last_counters()[0] == p.n_crystals * p.n_voxels * np.prod(sv) * np.prod(sc)
    g.close()
    ctx.close()


def test_a_batch_of_all_forms_equals_single_launches():
    """Rotated and unrotated detectors, few and many rays per entry, in one batch (a launch per form)."""
    ctx = sysmat_b200.Context(0)
    geos, opts, single = [], [], []
    for i in range(8):
        p = configs.tiny(seed=i, layers=1 + i % 3, rotated=bool(i & 1))
        if i & 2:
            p.sv = (2, 2, 2)
        g = sysmat_b200.Geometry(ctx, p)
        geos.append(g)
        opts.append(g.options())
        single.append(g.pe(opts=opts[-1]))
    outs = [torch.zeros(a.shape, dtype=torch.float32, device="cuda") for a in single]
    batch = sysmat_b200.PeBatch(ctx, geos, opts, [o.data_ptr() for o in outs], [o.shape[1] for o in outs])
    batch.run()
    torch.cuda.synchronize()
    for a, o in zip(single, outs):
        assert np.allclose(o.cpu().numpy(), a, rtol=1e-4, atol=1e-30)
    batch.close()
    for g in geos:
        g.close()
    ctx.close()
