"""The process-wide choices of kernel forms: what the library starts with, and that a test which changes them
leaves nothing to the next."""

import pytest

pytest.importorskip("torch")

from more_benchmarks_dc_ocean_b200 import autotune as T  # noqa: E402


@pytest.mark.parametrize("turn", ["first", "second"])
def test_defaults_in_force_and_not_left_changed(redi_lib, turn):
    assert T.get_tuning() == (64, 2, 8)
    assert T.get_gather_tracers() == (2, 4)
    assert T.get_tracer_group() == 2 and T.get_sweep_form() == 4 and T.get_flux_staged() == 0
    assert T.get_fold() == (0, 2, 0)
    T._apply((32, 4, 8))  # a choice without a gather form: sums in registers
    assert T.get_gather_tracers() == (2, 0)
    T.set_tracer_group(8)
    T.set_sweep_form(3)
    T.set_flux_staged(1)
    T.set_fold(T.FOLD_FP64, 1, 2)
