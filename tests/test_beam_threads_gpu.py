"""sm_beam_metrics called by several host threads at once, with rows of other lengths and
so other amounts of shared memory: every call succeeds and gives what it gives alone."""
import threading

import pytest

import sysmat_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(22000, 4100), (16000, 8192), (2047, 35)])
def test_calls_of_other_row_lengths_at_once(lengths):
    import torch
    odd = max(lengths) < 2048                          # unaligned rows: the other instantiation
    jobs = []
    for v in lengths * 2:
        a = torch.rand((40, (v + 3) // 4 * 4 + odd), device="cuda")
        mx = torch.empty(40, device="cuda")
        sm = torch.empty(40, dtype=torch.float64, device="cuda")
        ct = torch.empty(40, dtype=torch.int32, device="cuda")
        jobs.append((a, v, mx, sm, ct, torch.cuda.Stream()))
    torch.cuda.synchronize()
    codes = []

    def work(job):
        a, v, mx, sm, ct, stream = job
        for _ in range(4000):
            rc = sysmat_b200.lib().sm_beam_metrics(a.data_ptr(), 40, v, a.shape[1], 0.5, mx.data_ptr(), sm.data_ptr(),
                                                   ct.data_ptr(), None, 0, None, stream.cuda_stream)
            if rc != 0:
                codes.append((v, rc))
                return

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not codes
    for a, v, mx, sm, ct, _ in jobs:
        x = a[:, :v]
        assert torch.equal(mx, x.amax(1))
        assert torch.equal(ct, (x > 0.5 * mx[:, None]).sum(1, dtype=torch.int32))
        assert ((sm - x.double().sum(1)).abs() <= 1e-12 * sm).all()
