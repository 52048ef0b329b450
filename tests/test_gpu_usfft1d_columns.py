"""The adjoint along the height at the sizes where its walk up the columns can go
wrong, against the float64 restatement: more samples than cells, cells that no
sample reaches, the periodic wrap (no tilt: both ends of the samples reach the
same cells), partly filled blocks of columns.

Bound: as for the adjoint in the plane (float32 positions, short float32 sums):
2e-5."""
import math

import numpy as np
import pytest

from conftest import rel_l2
from oracle import np_tomo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n0,n1,rh,deth,tilt", [
    (130, 3, 32, 64, 30.0), (64, 2, 8, 200, 25.0), (33, 5, 120, 24, 61.3), (128, 1, 40, 80, 0.0),
    (20, 4, 26, 26, 3.0)])
def test_usfft1d_adj_vs_float64(cuda, n0, n1, rh, deth, tilt):
    import torch
    from tomocupy_b200.cfunc_usfft1d import cfunc_usfft1d
    rng = np.random.default_rng(n0)
    shape = (n1, deth // 2 + 1, n0)
    g = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    phi = math.pi / 2 + tilt / 180 * math.pi
    want = np_tomo.usfft1d_adj64(g.astype(np.complex128), float(np.float32(phi)), rh, deth)
    op = cfunc_usfft1d(rh, n1, n0, deth)
    f = torch.full((n1, rh, n0), float("nan"), device=cuda)
    op.adj(f, torch.as_tensor(g, device=cuda), phi, torch.cuda.current_stream())
    assert rel_l2(f.cpu().numpy(), want) < 2e-5
