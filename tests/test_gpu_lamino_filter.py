"""The two filters of the laminography chain -- the fused one (even chunk, axis a
whole number of pixels off the middle) and the padded one -- against the float64
restatement, and that changes of ``center`` and ``wfilter`` after construction
reach the next call.

Bound: the chain with the axis in the middle differs from float64 by 6e-6
(float32 positions and sums); 2e-5, as in test_gpu_lamino.py."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

NTHETA, DETH, DETW, RH, TILT = 27, 64, 64, 32, 30.0


def _data():
    rng = np.random.default_rng(8)
    return (rng.standard_normal((NTHETA, DETH, DETW)).astype(np.float32),
            (np.arange(NTHETA) * 2 * np.pi / NTHETA + 0.01).astype(np.float32))


def _object(center, ncproj):
    from tomocupy_b200 import global_vars
    from tomocupy_b200.global_vars import params
    from tomocupy_b200.reconstruction.backproj_lamfourier_parallel import \
        BackprojLamFourierParallel
    global_vars.reset(lamino_angle=TILT, reconstruction_algorithm="fourierrec",
                      nsino_per_chunk=8, nproj_per_chunk=ncproj, fbp_filter="shepp")
    params.n, params.nz, params.nproj, params.ncproj, params.ncz = DETW, DETH, NTHETA, ncproj, 8
    params.rh, params.center, params.theta, params.lamino_angle = RH, center, _data()[1], TILT
    return BackprojLamFourierParallel()


def _check(bp, data, center, wf, fused):
    from oracle import np_tomo
    assert (bp._fused() is not None) == fused
    want = np_tomo.rec_lam64(data, _data()[1], center, TILT, RH, wf)
    assert rel_l2(bp.rec_lam(data_on_gpu(data)).cpu().numpy(), want) < 2e-5


def data_on_gpu(data):
    import torch
    return torch.as_tensor(data, device="cuda")


@pytest.mark.parametrize("shift,ncproj,fused", [
    (0, 8, True), (3, 8, True), (-2, 10, True), (0.5, 8, False), (0, 9, False), (2.25, 7, False)])
def test_both_filters_vs_float64(cuda, shift, ncproj, fused):
    from oracle import np_tomo
    center = DETW / 2 + shift
    _check(_object(center, ncproj), _data()[0], center, np_tomo.calc_filter(4 * DETW, "shepp"),
           fused)


def test_changed_center_and_filter(cuda):
    from oracle import np_tomo
    data, wf = _data()[0], np_tomo.calc_filter(4 * DETW, "shepp")
    bp = _object(DETW / 2, 8)
    for shift, fused in ((0, True), (4, True), (1.5, False), (-1, True)):
        bp.center = DETW / 2 + shift
        _check(bp, data, bp.center, wf, fused)
    bp.wfilter.mul_(2)   # in place, then another tensor
    _check(bp, data, bp.center, 2 * wf, True)
    hann = np_tomo.calc_filter(4 * DETW, "hann")
    bp.wfilter = data_on_gpu(hann)
    _check(bp, data, bp.center, hann, True)
