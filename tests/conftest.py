"""Test configuration: markers and import paths.

`-m gpu` tests need a B200 and the built library libcgfd.so; those against the
reference's own runtime also its driver oracle/_ref/ref_wavesim, built from the
reference's sources (oracle/ref/Makefile), and are skipped without it;
`-m "not gpu"` tests run on
the CPU: the oracle against the reference's golden vectors, the host-side
pre-processing, and the C ABI's symbol table.
"""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (os.path.join(ROOT, "copara-cgfd3d_b200", "python"), os.path.join(ROOT, "oracle"),
          os.path.join(ROOT, "tests"), os.path.join(ROOT, "tests", "golden")):
    if p not in sys.path:
        sys.path.insert(0, p)


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """Tests that ask for the reference's driver (refio.run raises
    FileNotFoundError without it) are skipped where it was not built."""
    outcome = yield
    if outcome.excinfo is None or not issubclass(outcome.excinfo[0], FileNotFoundError):
        return
    import refio
    if not refio.available() and "ref_wavesim" in str(outcome.excinfo[1]):
        outcome.force_exception(pytest.skip.Exception(str(outcome.excinfo[1])))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and the built libraries")
    config.addinivalue_line("markers", "slow: longer full-size parity runs")


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    import fakecuda
    path = fakecuda.build(str(tmp_path_factory.mktemp("fakecuda")))
    if path is None:
        pytest.skip("nvcc and g++ are needed")
    return fakecuda.lib(path)


@pytest.fixture
def fake(fake_lib, monkeypatch):
    """The library on a CUDA runtime that lives on the host (tests/fakecuda)."""
    import cgfd
    fake_lib.fake_reset()
    monkeypatch.setattr(cgfd, "_lib", fake_lib)
    return fake_lib
