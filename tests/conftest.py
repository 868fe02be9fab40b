import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

GOLDEN = Path(__file__).resolve().parent / "golden"


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (sm_103a) and the built libcolagb")


@pytest.fixture
def golden():
    import numpy as np

    def load(name):
        return dict(np.load(GOLDEN / f"{name}.npz"))
    return load


@pytest.fixture
def kernels_of():
    """kernels_of(f) -> (f(), the names of the CUDA kernels it launched).  A profile may come back empty (the
    profiler's first use does): f, which has to be repeatable, is then run again."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    def run(f):
        for _ in range(4):
            torch.cuda.synchronize()
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                out = f()
                torch.cuda.synchronize()
            names = [e.key for e in prof.key_averages() if "colagb" in e.key]
            if names:
                return out, names
        pytest.skip("the profiler records no kernels here")
    return run


def cuda_available():
    import torch
    return torch.cuda.is_available()
