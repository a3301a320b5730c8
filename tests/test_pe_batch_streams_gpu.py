"""Two batches of other geometries at once, each on a stream of its own, between them all four
forms (few or many rays per entry, without or with rotated crystals): every matrix equals,
bit for bit, what the geometry gives alone."""
import numpy as np
import pytest

import sysmat_b200
from sysmat_b200 import configs

pytestmark = pytest.mark.gpu


def test_batches_on_two_streams():
    import torch
    ctx = sysmat_b200.Context(0)
    many_rotated = configs.tiny(seed=3, rotated=True)
    many_rotated.sv = (2, 2, 2)
    sets = [[configs.tiny(seed=i, layers=1 + i % 3, rotated=i == 4) for i in range(5)],
            [configs.two_plates_small(seed=8), configs.tiny(seed=9, layers=2), many_rotated,
             configs.sweep_small()[3]]]
    geos = [[sysmat_b200.Geometry(ctx, p) for p in params] for params in sets]
    want = [[g.pe() for g in gs] for gs in geos]
    outs = [[torch.empty(w.shape, device="cuda") for w in ws] for ws in want]
    batches = [sysmat_b200.PeBatch(ctx, gs, [g.options() for g in gs], [o.data_ptr() for o in os], [o.shape[1] for o in os])
               for gs, os in zip(geos, outs)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(5):
        for o in outs[0] + outs[1]:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(3):
            for b, s in zip(batches, streams):
                b.run(s.cuda_stream)
        torch.cuda.synchronize()
        for ws, os in zip(want, outs):
            for w, o in zip(ws, os):
                assert np.array_equal(o.cpu().numpy(), w)
    for b in batches:
        b.close()
    for g in geos[0] + geos[1]:
        g.close()
    ctx.close()
