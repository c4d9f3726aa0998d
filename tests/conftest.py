import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


# tests that run programs built from the reference sources (make -C oracle): where neither is there, there is nothing to run
REFERENCE_PROGRAMS = os.path.join(ROOT, "oracle", "_ref", "engine")
NEED_REFERENCE_PROGRAMS = ("test_gpu_engine_dropin.py", "test_reference_driver_resumes_from_a_checkpoint_the_fused_trainer_wrote")


def pytest_collection_modifyitems(config, items):
    import __graft_entry__ as entry
    if not os.path.isdir(REFERENCE_PROGRAMS) and entry.reference_dir() is None:
        skip = pytest.mark.skip(reason="neither oracle/_ref/engine nor the reference sources it is built from are here")
        for it in items:
            if any(n in it.nodeid for n in NEED_REFERENCE_PROGRAMS):
                it.add_marker(skip)
    try:
        import torch
        has_gpu = torch.cuda.is_available()
    except Exception:  # pragma: no cover
        has_gpu = False
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.fixture(autouse=True)
def _release_device_buffers():
    yield
    mod = sys.modules.get("tests.gpu_util")
    if mod is not None:
        mod.release()
