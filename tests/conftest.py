import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: long-running case")


@pytest.fixture(scope="session")
def oracle_lib():
    from oracle import oracle

    oracle.build()
    return oracle


@pytest.fixture(scope="session")
def redi_lib():
    from more_benchmarks_dc_ocean_b200 import build

    build.build()
    from more_benchmarks_dc_ocean_b200 import ocean_redi

    if not _tunables:
        _tunables.append(_tunables_now())
    return ocean_redi


# The process-wide choices of kernel forms as the library starts with them.
_tunables = []


def _tunables_now():
    from more_benchmarks_dc_ocean_b200 import autotune as T

    return (T.get_tuning(), T.get_gather_tracers(), T.get_tracer_group(), T.get_sweep_form(), T.get_flux_staged(),
            T.get_fold())


@pytest.fixture(autouse=True)
def _default_tunables():
    """Every test starts from the library's own choice of forms, whatever the ones before it left."""
    yield
    if _tunables and _tunables_now() != _tunables[0]:
        from more_benchmarks_dc_ocean_b200 import autotune as T

        shape, gather, group, sweep, staged, fold = _tunables[0]
        T.set_tuning(*shape)
        T.set_gather_tracers(*gather)
        T.set_tracer_group(group)
        T.set_sweep_form(sweep)
        T.set_flux_staged(staged)
        T.set_fold(*fold)
