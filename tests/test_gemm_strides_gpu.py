"""The BF16 GEMM's strides: rows that coincide, overlap or run backwards, k backwards or
apart, bases on and off 4 and 16 bytes, against an fp32 product of the same elements.
Tolerance 1e-4 of the row scale, as in test_gemm_gpu.py: fp32 accumulation in another
order, inputs identical."""
import pytest

import sysmat_b200

pytestmark = pytest.mark.gpu

STRIDES = [(0, 1), (8, 1), (5, 1), (-200, 1), (-203, 1), (208, 1), (1, -300), (300, 2), (0, 0), (3, 7)]


@pytest.mark.parametrize("base", [0, 1, 2, 8])
@pytest.mark.parametrize("sa", STRIDES)
def test_strides(sa, base):
    import torch
    torch.manual_seed(4)
    m, n, k = 150, 70, 130
    sb = STRIDES[(STRIDES.index(sa) * 3 + base) % len(STRIDES)]

    def operand(rows, s):
        low = min(0, (rows - 1) * s[0]) + min(0, (k - 1) * s[1])
        span = abs((rows - 1) * s[0]) + abs((k - 1) * s[1]) + 1
        start = (16 - low + 15) // 16 * 16 + base
        flat = torch.randn(start + span + 64, device="cuda").bfloat16()
        at = start + torch.arange(rows, device="cuda")[:, None] * s[0] + torch.arange(k, device="cuda")[None, :] * s[1]
        return flat, flat.data_ptr() + 2 * start, flat[at]

    keep_a, pa, a = operand(m, sa)
    keep_b, pb, b = operand(n, sb)
    c = torch.full((m, n), float("nan"), device="cuda")
    sysmat_b200.gemm_bf16(m, n, k, pa, sa, pb, sb, c.data_ptr(), n)
    torch.cuda.synchronize()
    want = a.float() @ b.float().T
    assert ((c - want).abs() / want.abs().amax(1, keepdim=True).clamp_min(1e-6)).max().item() <= 1e-4
