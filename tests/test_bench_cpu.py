"""What bench.py reports beside its measured times, with the measured calls stubbed out."""

import types

import pytest

torch = pytest.importorskip("torch")

import bench  # noqa: E402
from more_benchmarks_dc_ocean_b200 import autotune as T, inputs  # noqa: E402


def test_mixed_lines_try_the_default_gather_and_leave_the_forms_alone(redi_lib, monkeypatch):
    """The mixed-precision lines choose among shapes that include the library's default gather, and the
    process goes on with the forms it had."""
    seen = []

    def tune(dp, redi, candidates, **_):
        seen.append(list(candidates))
        T._apply(candidates[0])
        return {"best": candidates[0], "ms": {}}

    def tune_group(*_, **__):
        T.set_tracer_group(8)
        return {"best": (8, 2), "ms": {}}

    p = inputs.make_problem(12, 10, 4, seed=1)
    monkeypatch.setattr(T, "tune", tune)
    monkeypatch.setattr(T, "tune_tracer_group", tune_group)
    monkeypatch.setattr(bench, "_time_steps", lambda *a: 1.0)
    monkeypatch.setattr(inputs, "config3", lambda: p)
    monkeypatch.setattr(redi_lib, "make_redi", lambda *a: types.SimpleNamespace(destroy=lambda: None))
    monkeypatch.setattr(redi_lib, "to_device", lambda *a: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: None)
    before = (T.get_tuning(), T.get_gather_tracers(), T.get_tracer_group())
    bench._mixed_batched(types.SimpleNamespace(steps=3), p, None, None, 1.0)
    assert (T.get_tuning(), T.get_gather_tracers(), T.get_tracer_group()) == before
    default = before[0] + (before[1][1],)
    assert len(seen) == 2 and all(default in c for c in seen), seen


def test_every_kernel_id_has_a_name(redi_lib):
    assert len(bench.KERNEL_NAMES) == redi_lib.lib().redi_b200_kernel_count()


@pytest.mark.parametrize("launches", [False, True])
def test_the_batch_line_names_the_form_it_timed(launches):
    ps = [inputs.make_problem(12, 10, 4, seed=1)]
    kid, kernel, words = bench._batch_form(launches)
    block = bench._domains_config_block(ps, types.SimpleNamespace(precision="fp64"), 1, "plain FP64", launches)
    assert words in block["workload"] and ("persistent" in block["workload"]) == (not launches)
    assert bench.KERNEL_NAMES[kid] == ("k_batch_gate" if launches else "k_domain_persistent")
    assert ("persistent" in kernel) == (not launches)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_kernel_bytes_of_a_step(precision):
    """The kernels of a whole step: the coefficients are written once, by the sweep with fluxes; the gather's
    launches, however many, read and write every tracer once."""
    p = inputs.make_problem(30, 20, 6, n_passive=7, seed=2)
    by = lambda name, n=1.0: bench.kernel_bytes(p, bench.KERNEL_NAMES.index(name), precision, n)  # noqa: E731
    surf = ((p.nx + 1) * p.ny + p.nx * (p.ny + 1)) * (2 * p.nz + 2) * (32 if precision == "fp64" else 24)
    sweep = by("k_sweep_flux" if precision == "fp64" else "k_mixed_sweep_flux")
    assert surf < sweep < 1.2 * surf
    cells = p.nx * p.ny
    for launches in (1, 2, 5):
        assert launches * by("k_cell_gather", launches) == pytest.approx(16 * cells * p.nz * p.ntr + 8 * cells * launches)


def test_measured_traffic_is_of_kernels_that_a_step_launches():
    assert set(bench._ncu_traffic()) == {"k_column_recon", "k_sweep_flux", "k_cell_gather"}
