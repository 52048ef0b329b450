"""Vo's ring removal beside a pixel without signal (flat and dark zero: a column of
NaN, 0/0, or of infinities, x/0), against the oracle with medians that rank NaN
last, as NumPy's and CuPy's sorts do.  Tolerance: as in test_gpu_stripe_vo.py."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _median_nan_last(a, size):
    """scipy.ndimage.median_filter (mode reflect) along the one axis of size > 1."""
    ax = int(np.argmax(size))
    w = size[ax]
    pad = [(0, 0)] * a.ndim
    pad[ax] = (w // 2, w // 2)
    win = np.lib.stride_tricks.sliding_window_view(np.pad(a, pad, mode="symmetric"), w, axis=ax)
    return np.sort(win, axis=-1)[..., w // 2]


@pytest.mark.parametrize("nproj,nz,ni,la,sm,bad", [
    (40, 2, 300, 31, 11, {50: np.nan}), (64, 1, 420, 61, 21, {130: np.nan, 131: np.nan, 300: np.nan}),
    (30, 2, 140, 15, 5, {0: np.nan, 139: np.nan}), (48, 1, 200, 21, 9, {60: np.inf, 150: np.nan})])
def test_columns_without_signal(cuda, monkeypatch, nproj, nz, ni, la, sm, bad):
    import scipy.ndimage as ndi
    from oracle import np_tomo
    from tomocupy_b200.processing.remove_stripe import remove_all_stripe
    rng = np.random.default_rng(ni)
    data = (1 + 0.1 * np.sin(np.arange(nproj) / 7)[:, None, None]
            + 0.02 * rng.standard_normal((nproj, nz, ni))).astype(np.float32)
    for x, v in bad.items():
        data[:, :, x] = v
    monkeypatch.setattr(ndi, "median_filter", _median_nan_last)
    with np.errstate(invalid="ignore"):
        want = np_tomo.remove_all_stripe(data, 3.0, la, sm)
    got = remove_all_stripe(torch.as_tensor(data, device=cuda), 3.0, la, sm).cpu().numpy()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    assert rel_l2(np.nan_to_num(got), np.nan_to_num(want)) < 1e-5
