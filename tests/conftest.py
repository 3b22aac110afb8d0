import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "oracle"))

import oracle as O   # noqa: E402

_not_compared = []


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


# A comparison with the oracle cannot be made where its library is absent and there are no reference sources to build it
# from: such a test is skipped, and the summary says how many there were.  With the sources at hand (AV1GPU_REF) a missing
# library is a failure.
def _without_oracle(item, ex):
    if os.path.isdir(os.path.join(os.environ.get("AV1GPU_REF", ""), "av1core", "src")):
        raise ex
    _not_compared.append(item.nodeid)
    pytest.skip("oracle library absent, no reference sources to build it from")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    try:
        return (yield)
    except O.OracleMissing as ex:
        _without_oracle(item, ex)


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    try:
        return (yield)
    except O.OracleMissing as ex:
        _without_oracle(item, ex)


def pytest_terminal_summary(terminalreporter):
    if _not_compared:
        terminalreporter.write_line("%d tests skipped: the oracle library (oracle/_ref/liboracle.so) is absent, so nothing was "
                                    "compared with it or with av1core" % len(_not_compared))


@pytest.fixture(scope="session")
def enc():
    from av1gpu_b200 import Encoder
    e = Encoder(0)
    yield e
    e.close()
