"""The BF16 GEMM with waits of a few polls, so that any of its roles may be the one whose
wait runs out, with copies and MMAs of the others in flight: the error word tells, a launch
that reports none is correct, and the next launch with the default limit is correct."""
import pytest

import sysmat_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1, 2, 4, 16, 64, 512])
@pytest.mark.parametrize("m,n,k,pitch", [
    (128, 256, 256, 0),      # one tile whose loads need no slot twice
    (384, 256, 256, 0),      # B kept
    (384, 512, 640, 0),      # the ring wraps
    (200, 300, 200, 3),      # the loader warps
])
def test_any_wait_may_run_out(m, n, k, pitch, limit):
    import torch
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k + pitch, device="cuda").bfloat16()
    b = torch.randn(n, k, device="cuda").bfloat16()
    ref = a[:, :k].float() @ b.float().T
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def launch():
        c = torch.full((m, n), float("nan"), device="cuda")
        err.zero_()
        sysmat_b200.gemm_bf16(m, n, k, a.data_ptr(), (k + pitch, 1), b.data_ptr(), (k, 1), c.data_ptr(), n,
                              error=err.data_ptr())
        torch.cuda.synchronize()
        return c, int(err.item())

    def good(c):
        # fp32 accumulation in another order, inputs identical: 1e-4 of the row scale as in test_gemm_gpu.py
        return ((c - ref).abs() / ref.abs().amax(1, keepdim=True)).max().item() <= 1e-4

    for _ in range(10):
        sysmat_b200.tc_wait_limit(limit)
        try:
            c, e = launch()
        finally:
            sysmat_b200.tc_wait_limit(-1)
        assert e in (0, 1) and (e == 1 or good(c))
        c, e = launch()
        assert e == 0 and good(c)
