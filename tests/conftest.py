import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a B200 (runs the CUDA engine)")
    config.addinivalue_line("markers", "slow: long CPU oracle runs")


REF_DIR = os.path.join(ROOT, "oracle", "_ref")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """Tests that run the reference's own programs need its rebuild (make -C oracle
    ref, where its sources are); without it they are skipped, with that reason."""
    try:
        return (yield)
    except FileNotFoundError as e:
        missing = os.path.realpath(str(e.filename or ""))
        if os.path.dirname(missing) == os.path.realpath(REF_DIR) and not os.path.exists(missing):
            pytest.skip(f"reference program not built: oracle/_ref/{os.path.basename(missing)}")
        raise


@pytest.fixture(scope="session")
def orc():
    import oracle
    oracle.lib()
    return oracle


@pytest.fixture(scope="session")
def ps():
    """The engine package; on a GPU test run the CUDA library must load."""
    import cuda_pspin_b200
    cuda_pspin_b200.load_library()
    return cuda_pspin_b200
