"""GPU check of the packed filter banks of the Fourier-wavelet ring removal
(src/tomocupy/processing/remove_stripe.py:51-293) against the oracle's
restatement at the sizes where their tiles end: an odd count of rows (the last
pair holds one row, or two of different sinograms), widths around the 4- and
8-output groups and the 64-column tiles, bands shorter than the filters, a row
too wide for 48 KB of shared memory, levels large enough for the full count of
outputs per thread and two pairs of rows per block.  The wavelet stages keep the oracle's float32
operation order; the band damping differs by less than 1e-6 (rel-L2, see
test_gpu_stripe.py), which is the tolerance."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import np_tomo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nproj,nz,n,level,wname", [
    (24, 1, 33, 2, "sym16"), (25, 3, 64, 1, "sym16"), (180, 3, 127, 4, "sym16"),
    (91, 3, 130, 3, "db5"), (57, 1, 1021, 5, "sym16"), (24, 3, 97, 3, "haar"),
    (40, 2, 2050, 7, "sym16"), (16, 1, 7000, 2, "sym16"), (33, 5, 63, 2, "db5"),
    (401, 3, 1290, 2, "sym16"), (700, 2, 1026, 2, "db5"), (420, 3, 1300, 1, "haar"),
])
def test_fw_tiles(cuda, nproj, nz, n, level, wname):
    from tomocupy_b200.processing import wavelets
    from tomocupy_b200.processing.remove_stripe import remove_stripe_fw
    rng = np.random.default_rng(nproj + n)
    data = (1 + 0.1 * rng.standard_normal((nproj, nz, n))).astype(np.float32)
    out = remove_stripe_fw(torch.as_tensor(data, device=cuda), 1.0, wname, level)
    want = np_tomo.remove_stripe_fw(data, 1.0, level, wavelets.filter_bank(wname))
    assert rel_l2(out.cpu().numpy(), want) < 1e-6
