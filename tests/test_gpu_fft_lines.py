"""fourierrec's inverse transform of widths that are no powers of two: the
mixed-radix lines at every radix (3 .. 18) and count of stages, and cuFFT on the
transposed columns, against one full cuFFT transform of the same grid.

Bound: each stage rounds a value a few times (2^-24 relative), four stages in
either transform: below 1e-6 of the result's norm."""
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


# the radices of 2n: 17 4 | 9 8 | 11 8 | 6 16 | 13 8 | 9 3 4 | 5 5 4 | 10 16 | 7 7 4 | 14 16 |
# 18 16 | 15 4 16 .. | 15 6 16 | 15 3 16 4 | 17 18 16; a prime above 17 at 38 and 1058
@pytest.mark.parametrize("n,nproj,nz", [
    (34, 5, 3), (36, 7, 1), (44, 9, 2), (48, 5, 5), (52, 4, 1), (54, 6, 2), (50, 3, 4), (80, 5, 2),
    (98, 4, 1), (112, 6, 3), (144, 5, 2), (240, 8, 2), (720, 6, 1), (1440, 5, 1), (2448, 6, 1),
    (38, 5, 3), (1058, 5, 1)])
def test_lines_vs_full_transform(cuda, monkeypatch, n, nproj, nz):
    import torch
    rng = np.random.default_rng(n)
    g = torch.as_tensor(rng.standard_normal((nz, nproj, n, 2)).astype(np.float32), device=cuda)
    theta = torch.as_tensor((np.arange(nproj) * np.pi / nproj + 0.01).astype(np.float32),
                            device=cuda)
    args = (monkeypatch, cuda, n, nproj, nz, g, theta)
    want = _run(*args, {"TCB_FOURIERREC_FULL_FFT2D": "1"})
    assert rel_l2(_run(*args, {}), want) < 1e-6
    assert rel_l2(_run(*args, {"TCB_FOURIERREC_FFT": "cufft"}), want) < 1e-6


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
