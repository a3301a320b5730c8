"""sm_beam_metrics at the row lengths where its kernels change (short unaligned rows, rows
kept in shared memory, rows held in registers, long rows) and at their tails, against the
same quantities by torch: maximum, mask, counts and MPXI exactly, sums to 1e-12."""
import pytest

import sysmat_b200

pytestmark = pytest.mark.gpu


def check(rows, voxels, ld, ldm, with_mask, with_mpxi):
    import torch
    torch.manual_seed(rows + voxels)
    a = torch.randn((rows, ld), device="cuda").mul_(2.5).exp_()
    a[::7] = 0.0
    a[1::11, :voxels] *= -1.0
    a[:, voxels:] = float("inf")                       # the pitch is not part of the row
    mx = torch.empty(rows, device="cuda")
    sm = torch.empty(rows, dtype=torch.float64, device="cuda")
    ct = torch.empty(rows, dtype=torch.int32, device="cuda")
    mask = torch.full((rows, ldm), 7, dtype=torch.int8, device="cuda") if with_mask else None
    mpxi = torch.full((voxels,), 7, dtype=torch.int32, device="cuda") if with_mpxi else None
    sysmat_b200._check(sysmat_b200.lib().sm_beam_metrics(
        a.data_ptr(), rows, voxels, ld, 0.05, mx.data_ptr(), sm.data_ptr(), ct.data_ptr(),
        mask.data_ptr() if with_mask else None, ldm, mpxi.data_ptr() if with_mpxi else None,
        torch.cuda.current_stream().cuda_stream))
    x = a[:, :voxels]
    want = x.amax(1)
    thr = torch.where(want > 0, want * torch.tensor(0.05, device="cuda"), torch.ones_like(want))
    assert torch.equal(mx, want)
    for r0 in range(0, rows, 4096):
        part = slice(r0, r0 + 4096)
        m = x[part] > thr[part, None]
        ref = x[part].double()
        assert ((sm[part] - ref.sum(1)).abs() <= 1e-12 * ref.abs().sum(1)).all()
        assert torch.equal(ct[part], m.sum(1, dtype=torch.int32))
        if with_mask:
            assert torch.equal(mask[part, :voxels], m.to(torch.int8)) and (mask[part, voxels:] == 7).all()
    if with_mpxi:
        assert torch.equal(mpxi, sum((x[r0:r0 + 4096] > thr[r0:r0 + 4096, None]).sum(0, dtype=torch.int32)
                                     for r0 in range(0, rows, 4096)))


@pytest.mark.parametrize("voxels", [1, 3, 33, 257, 2047, 2048, 2049, 8188, 8192, 8195, 12001, 16384, 16388, 22999, 23004])
def test_row_lengths(voxels):
    up = (voxels + 3) // 4 * 4
    check(613, voxels, up, up, True, True)             # aligned
    check(300, voxels, up + 1, up + 3, True, True)     # unaligned rows and masks
    check(5, voxels, up + 4, up, False, True)
    check(2, voxels, up, up + 4, True, False)


def test_counts_of_many_rows_per_block():
    check(76500, 8192, 8192, 8192, False, True)        # more rows per block than a byte counts
