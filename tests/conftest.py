import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "nitroozk-stwo_b200"), os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: long-running case")


@pytest.fixture(scope="module", autouse=True)
def fft_splits_by_size():
    """Modules that install FFT pass splits leave none behind."""
    yield
    backend = sys.modules.get("gpustark.backend")
    if backend is not None and os.path.exists(backend.L.LIB_PATH):
        backend.GpuBackend.fft_reset_tuning()
