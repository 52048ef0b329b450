"""fourierrec's inverse transform of widths that are no powers of two: cuFFT on the
rows and then on the kept columns, transposed or within the grid, against one full
cuFFT transform of the same grid.

Bound: a transform of these lengths rounds a value a few times at each of its
stages (2^-24 relative): below 1e-6 of the result's norm."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(monkeypatch, cuda, n, nproj, nz, g, theta, env):
    import torch
    from tomocupy_b200 import _lib
    from tomocupy_b200.cfunc_fourierrec import cfunc_fourierrec
    for k in ("TCB_FOURIERREC_FFT", "TCB_FOURIERREC_FULL_FFT2D"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    op = cfunc_fourierrec(nproj, nz, n, theta)
    op.set_gridding(_lib.GRID_FP32)
    f = torch.full((nz, n, n, 2), float("nan"), device=cuda)
    op.backprojection(f, g.clone(), torch.cuda.current_stream())
    return f.cpu().numpy()


# fewer than 640 columns in all (within the grid); beside the 32 x 32 and 64 x 32
# tiles; one, several and a remainder of pairs per block; primes of 2n up to 1223
@pytest.mark.parametrize("n,nproj,nz", [
    (34, 5, 3), (240, 8, 2), (319 * 2, 5, 1), (640, 4, 1), (38, 5, 20), (66, 3, 10), (98, 4, 8),
    (300, 5, 40), (720, 6, 5), (1058, 5, 9), (2446, 3, 1), (2448, 6, 2)])
def test_columns_vs_full_transform(cuda, monkeypatch, n, nproj, nz):
    import torch
    rng = np.random.default_rng(n)
    g = torch.as_tensor(rng.standard_normal((nz, nproj, n, 2)).astype(np.float32), device=cuda)
    theta = torch.as_tensor((np.arange(nproj) * np.pi / nproj + 0.01).astype(np.float32),
                            device=cuda)
    args = (monkeypatch, cuda, n, nproj, nz, g, theta)
    want = _run(*args, {"TCB_FOURIERREC_FULL_FFT2D": "1"})
    assert rel_l2(_run(*args, {}), want) < 1e-6


@pytest.mark.parametrize("n,nz", [(128, 5), (256, 12)])
def test_columns_of_power_of_two_widths(cuda, monkeypatch, n, nz):
    """cuFFT's route where the library's own transform is the usual one."""
    import torch
    g = torch.randn((nz, 30, n, 2), generator=torch.Generator(device=cuda).manual_seed(n),
                    device=cuda)
    theta = torch.as_tensor((np.arange(30) * np.pi / 30 + 0.01).astype(np.float32), device=cuda)
    args = (monkeypatch, cuda, n, 30, nz, g, theta)
    assert rel_l2(_run(*args, {"TCB_FOURIERREC_FFT": "cufft"}), _run(*args, {})) < 1e-6


def test_little_memory(cuda):
    """A handle is created as soon as what it cannot do without fits (the copy for
    the columns is given up), and gives the same images.  2n = 4 * 1223, for which
    cuFFT takes a workspace larger than the grid."""
    import torch
    from tomocupy_b200 import _lib
    from tomocupy_b200.cfunc_fourierrec import cfunc_fourierrec
    n, nproj, nz = 2446, 8, 8
    theta = torch.as_tensor((np.arange(nproj) * np.pi / nproj + 0.01).astype(np.float32),
                            device=cuda)
    g = torch.randn((nz, nproj, n, 2), generator=torch.Generator(device=cuda).manual_seed(1),
                    device=cuda)
    f, gc = torch.empty((nz, n, n, 2), device=cuda), torch.empty_like(g)

    def run(budget=None):
        """Bytes that a handle takes where `budget` are free (None: it is refused)."""
        torch.cuda.empty_cache()
        hold = None
        if budget is not None:
            hold = torch.empty(torch.cuda.mem_get_info()[0] - budget, dtype=torch.uint8,
                               device=cuda)
        before = torch.cuda.mem_get_info()[0]
        try:
            op = cfunc_fourierrec(nproj, nz, n, theta)
        except _lib.TcbError:
            return None
        finally:
            used = before - torch.cuda.mem_get_info()[0]
            del hold
            torch.cuda.empty_cache()
        gc.copy_(g)
        op.backprojection(f, gc, torch.cuda.current_stream())
        torch.cuda.synchronize()
        op.free()
        return used

    mb = 1 << 20
    lo, hi = nz * 4 * n * n * 8, run() + 64 * mb
    want = f.cpu().numpy()
    while hi - lo > 48 * mb:
        mid = (lo + hi) // 2 // mb * mb
        if run(mid) is None:
            lo = mid
        else:
            hi = mid
    assert hi - run(hi) < 160 * mb
    assert rel_l2(f.cpu().numpy(), want) < 1e-6
