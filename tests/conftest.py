import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def orc():
    """The CPU oracle (test infrastructure), built on first use."""
    from oracle import oracle
    oracle.build()
    return oracle


@pytest.fixture(scope="session")
def model_dir(tmp_path_factory):
    d = os.environ.get("WICK_SYNTH_CACHE") or str(tmp_path_factory.mktemp("wick_models"))
    os.makedirs(d, exist_ok=True)
    return d


@pytest.fixture(scope="session")
def cuda_lib():
    """The product library; building needs nvcc, running needs a GPU."""
    from wick_b200 import _lib, build
    build.build()
    return _lib.load()


@pytest.fixture
def cuda_core_weight(cuda_lib, monkeypatch):
    """Makes operator weights whose products stay on the CUDA cores, to compare the tensor-core kernels with (a plain weight's
    product of more than 8 columns is one of them itself)."""
    def make(dtype, raw, m, k):
        from wick_b200 import ops
        with monkeypatch.context() as mp:
            mp.setenv("WICK_CUDA_PREFILL", "exact-cuda-cores")
            return ops.QuantWeight(dtype, raw, m, k)
    return make
