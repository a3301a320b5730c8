"""The BF16 GEMM's ways of loading (TMA, shifted rows, gathered columns, B's tile kept in
shared memory), its tile widths, and its ragged edges, against an fp32 product of the same
bf16 inputs.  Tolerance 1e-4 of the row scale, as in test_gemm_gpu.py: fp32 accumulation
in another order, inputs identical."""
import pytest

import sysmat_b200

pytestmark = pytest.mark.gpu


def operand(rows, k, layout, torch):
    """(tensor to keep, pointer, strides, values [rows][k])."""
    if layout == "t":                                             # k strided
        x = torch.randn(k, rows, device="cuda").bfloat16()
        return x, x.data_ptr(), (1, rows), x.t()
    pad = {"c": 0, "odd": 0, "pad": 3, "pitch": 8 - k % 8}[layout]
    off = 1 if layout == "odd" else 0                             # base off 4 and 16 bytes
    flat = torch.randn(rows * (k + pad) + off, device="cuda").bfloat16()
    x = flat[off:].view(rows, k + pad)
    return flat, x.data_ptr(), (k + pad, 1), x[:, :k]


@pytest.mark.parametrize("m,n,k,la,lb", [
    (1, 1, 1, "c", "c"), (127, 63, 64, "c", "c"), (129, 65, 63, "odd", "c"), (130, 257, 65, "pad", "odd"),
    (257, 300, 129, "t", "pitch"), (40, 513, 200, "pitch", "t"), (200, 40, 33, "odd", "t"),
    (384, 40000, 256, "c", "c"),       # B kept, a second, narrower panel of tiles
    (2304, 4100, 250, "pitch", "pitch"), (640, 9000, 257, "pitch", "c"), (700, 9000, 319, "odd", "odd"),
])
def test_every_way_of_loading(m, n, k, la, lb):
    import torch
    torch.manual_seed(m + n + k)
    keep_a, pa, sa, a = operand(m, k, la, torch)
    keep_b, pb, sb, b = operand(n, k, lb, torch)
    ld = n + (n % 3)
    c0 = torch.randn(m, ld, device="cuda")
    c = c0.clone()
    scale, bias = torch.rand(m, device="cuda") + 0.5, torch.randn(n, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    sysmat_b200.gemm_bf16(m, n, k, pa, sa, pb, sb, c.data_ptr(), ld, row_scale=scale.data_ptr(), bias=bias.data_ptr(),
                          accumulate=True, error=err.data_ptr())
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = scale[:, None] * (a.float() @ b.float().T) + bias + c0[:, :n]
    assert ((c[:, :n] - ref).abs() / ref.abs().amax(1, keepdim=True).clamp_min(1e-6)).max().item() <= 1e-4
    assert torch.equal(c[:, n:], c0[:, n:])
    plain = torch.full((m, n), float("nan"), device="cuda")
    sysmat_b200.gemm_bf16(m, n, k, pa, sa, pb, sb, plain.data_ptr(), n)
    torch.cuda.synchronize()
    want = a.float() @ b.float().T
    assert ((plain - want).abs() / want.abs().amax(1, keepdim=True).clamp_min(1e-6)).max().item() <= 1e-4
