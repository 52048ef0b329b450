import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and the built library")


def rel_l2(a, b):
    import numpy as np
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU test selected but no CUDA device is available")
    return torch.device("cuda")


@pytest.fixture(scope="session")
def ref():
    """The reference CUDA build (oracle/_ref) driven through oracle.refglue.  Without
    the reference's sources it cannot be built, and the tests that compare with it
    are skipped; the float64 and NumPy restatements cover the same operators."""
    from oracle import refglue
    if not refglue.available():
        pytest.skip("oracle/_ref is not built: run `make -C oracle` (needs the reference sources)")
    return refglue


@pytest.fixture(params=["auto", "tensor"])
def gridding(request, monkeypatch):
    """fourierrec's gridding in the drivers: as the automatic rule chooses it (fp32
    registers at the few slices of a test), and on the tensor cores with streamed
    weights, which the rule takes for larger chunks."""
    if request.param == "tensor":
        from tomocupy_b200.pipeline import SinoPipeline
        choose = SinoPipeline._set_gridding

        def tensor(self, gridding, precision):
            return choose(self, "tensor_stream" if precision == "mixed" else "tensor_fp32",
                          precision)
        monkeypatch.setattr(SinoPipeline, "_set_gridding", tensor)
    return request.param


class TorchCuFFT:
    """Real FFTs through cuFFT (torch.fft on the GPU), the library that the
    reference's cupy.fft calls, with NumPy's types (float32 <-> complex64,
    float64 <-> complex128) and normalisation; a drop-in ``fft`` provider for
    the oracle's ring-removal restatements."""

    @staticmethod
    def rfft(a, axis=-1):
        import numpy as np
        import torch
        x = torch.as_tensor(np.ascontiguousarray(a), device="cuda")
        return torch.fft.rfft(x, dim=axis).cpu().numpy()

    @staticmethod
    def irfft(a, n, axis=-1):
        import numpy as np
        import torch
        x = torch.as_tensor(np.ascontiguousarray(a), device="cuda")
        return torch.fft.irfft(x, n=n, dim=axis).cpu().numpy()
