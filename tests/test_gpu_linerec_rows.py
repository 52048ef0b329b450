"""The one-row-per-slice line backprojection of tomography against the bilinear
kernel (plain staging), bit for bit: widths beside the 32 x 8 tiles, slice
counts beside the groups of 8 and 4, angle counts beside the 16 of a stage, row
offsets, rows past 256 (where v - 1e-5 rounds to v), and values that are not
finite (a slice takes the sum of its neighbour row's samples times zero)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nproj,nz,ncz,sz,bad", [
    (64, 33, 8, 8, 0, False), (52, 16, 9, 9, 0, False), (100, 17, 12, 12, 0, True),
    (132, 5, 300, 13, 250, True), (68, 48, 20, 3, 16, False), (96, 1, 2, 2, 0, True),
    (64, 20, 520, 16, 504, False), (200, 31, 1, 1, 0, False)])
def test_rows_equal_bilinear(cuda, monkeypatch, n, nproj, nz, ncz, sz, bad):
    import torch
    from tomocupy_b200.cfunc_linerec import cfunc_linerec
    g = torch.Generator(device=cuda).manual_seed(n)
    data = torch.randn((nz, nproj, n), generator=g, device=cuda)
    if bad:
        data[nz // 2, 0, n // 3] = math.inf
        data[nz - 1, nproj // 2, n // 2] = math.nan
    th = torch.as_tensor((np.arange(nproj) * math.pi / nproj + 0.01).astype(np.float32),
                         device=cuda)
    op = cfunc_linerec(nproj, nz, n, nproj, ncz)
    init = torch.randn((ncz, n, n), generator=g, device=cuda)
    rows, full = init.clone(), init.clone()
    stream = torch.cuda.current_stream()
    op.backprojection(rows, data, th, math.pi / 2, sz, stream)
    monkeypatch.setenv("TCB_LINEREC_TMA", "0")
    op.backprojection(full, data, th, math.pi / 2, sz, stream)
    assert not op.timed_out()
    assert torch.equal(rows.isnan(), full.isnan())
    assert torch.equal(rows.nan_to_num(0.0), full.nan_to_num(0.0))


def test_rows_beside_a_sum_that_overflows(cuda, monkeypatch):
    """A slice next to one whose finite samples add up to infinity stays finite."""
    import torch
    from tomocupy_b200.cfunc_linerec import cfunc_linerec
    n, nproj, nz = 64, 40, 12
    data = torch.randn((nz, nproj, n), generator=torch.Generator(device=cuda).manual_seed(3),
                       device=cuda)
    data[5] = 2e37
    th = torch.as_tensor((np.arange(nproj) * math.pi / nproj + 0.01).astype(np.float32),
                         device=cuda)
    op = cfunc_linerec(nproj, nz, n, nproj, nz)
    rows, full = (torch.zeros((nz, n, n), device=cuda) for _ in range(2))
    stream = torch.cuda.current_stream()
    op.backprojection(rows, data, th, math.pi / 2, 0, stream)
    monkeypatch.setenv("TCB_LINEREC_TMA", "0")
    op.backprojection(full, data, th, math.pi / 2, 0, stream)
    assert torch.isinf(full[5]).any() and torch.isfinite(full[[4, 6]]).all()
    assert torch.equal(rows, full)
