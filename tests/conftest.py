import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


def pytest_collection_modifyitems(items):
    """The VapourSynth plugin and its headless host are built where the SDK's
    header is at hand; without them their tests are skipped, as the AviSynth+
    ones are."""
    lib = os.path.join(ROOT, "neo_fft3d_b200", "lib")
    if all(os.path.exists(os.path.join(lib, f)) for f in ("libfft3d_vshost.so", "libneo_fft3d_vs.so")):
        return
    for item in items:
        if item.path.name in ("test_plugin.py", "test_plugin_formats.py"):
            item.add_marker(pytest.mark.skip(reason="VapourSynth host or plugin not built"))


def cuda_available() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def gpu():
    if not cuda_available():
        pytest.skip("no CUDA device")
    return 0
