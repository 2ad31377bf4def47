"""The tuner's choices, against a library that only counts launches and their time."""

import json
import types

import pytest

torch = pytest.importorskip("torch")

from more_benchmarks_dc_ocean_b200 import autotune, ocean_redi as R  # noqa: E402


class FakeLib:
    """The tuning, profiling and gather-form entry points over a table of kernel times.

    ``gather(form, ntr)`` gives the gather launches of one redi_apply_flux and the ms each takes."""

    def __init__(self, ntr, gather):
        self.ntr, self.gather = ntr, gather
        self.shape, self.form, self.n = (64, 2, 8), 4, 2
        self.kt, self.kc = [0.0] * 18, [0] * 18
        for name in ("set_tuning", "get_tuning", "set_gather_tracers", "get_gather_tracers", "profile_begin",
                     "profile_end", "kernel_count"):
            method = getattr(self, "_" + name)
            setattr(self, "redi_b200_" + name, lambda *a, m=method: m(*a))

    def _set_tuning(self, *shape):
        self.shape = shape
        return 0

    def _get_tuning(self, *out):
        for o, v in zip(out, self.shape):
            o._obj.value = v
        return 0

    def _set_gather_tracers(self, n, form):
        self.n, self.form = n, form
        return 0

    def _get_gather_tracers(self, out):
        out._obj.value = self.form
        return self.n

    def _kernel_count(self):
        return len(self.kt)

    def _profile_begin(self):
        self.kt, self.kc = [0.0] * 18, [0] * 18
        return 0

    def _profile_end(self, kt, kc, n):
        kt[:], kc[:] = self.kt, self.kc
        return 0

    def apply_flux(self, *_):
        launches, ms = self.gather(self.form, self.ntr)
        self.kt[3] += launches * ms
        self.kc[3] += launches
        self.kt[4] += 1.0
        self.kc[4] += 1


@pytest.fixture
def fake(monkeypatch, tmp_path):
    def make(ntr, gather):
        lib = FakeLib(ntr, gather)
        monkeypatch.setenv("REDI_B200_TUNING_CACHE", str(tmp_path / "tuning.json"))
        monkeypatch.setattr(R, "lib", lambda: lib)
        monkeypatch.setattr(R, "redi_calc_coeffs", lambda *a: 0)
        monkeypatch.setattr(R, "redi_apply_flux", lib.apply_flux)
        monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
        monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "fake")
        dp = types.SimpleNamespace(grid=types.SimpleNamespace(nx_total=20, ny_total=20), metrics=None, eos=None, dt=1.0,
                                   khtr_u_ext=None, khtr_v_ext=None, bc=None,
                                   ms=types.SimpleNamespace(nz_ml=10, tracers=[None] * ntr,
                                                            h_layer=types.SimpleNamespace(device="fake")))
        return lib, dp

    return make


@pytest.mark.parametrize("ntr", [2, 6, 34])
def test_forms_are_ranked_by_the_call(fake, ntr):
    """A launch of the row gather folds up to four pairs of tracers, one of the other forms a single pair:
    what counts is the time of all of a call's launches."""
    pairs = (ntr + 1) // 2
    lib, dp = fake(ntr, lambda form, n: (-(-pairs // 4), 0.8 * pairs / -(-pairs // 4)) if form == 4 else (pairs, 1.0))
    res = autotune.tune(dp, types.SimpleNamespace(precision=0), candidates=[(64, 2, 8, 3), (64, 2, 8, 4)], use_cache=False)
    assert res["best"] == (64, 2, 8, 4) and lib.form == 4, res
    assert res["ms"]["64x2/ch8/rows"] == pytest.approx(0.8 * pairs + 1.0)


def test_choices_of_an_older_set_of_forms_are_not_taken_up(fake, tmp_path):
    """An entry stored before the row gather was known (three or four numbers) is timed anew, and the new
    choice is found again."""
    lib, dp = fake(2, lambda form, n: (1, 1.0 if form == 4 else 2.0))
    for old in ([64, 2, 8], [64, 2, 8, 3]):
        (tmp_path / "tuning.json").write_text(json.dumps({"fake|small|nz10|ntr2|p0": old}))
        lib.form = 4
        res = autotune.tune(dp, types.SimpleNamespace(precision=0), candidates=[(64, 2, 8, 3), (64, 2, 8, 4)])
        assert not res["cached"] and res["best"] == (64, 2, 8, 4) and lib.form == 4, res
        lib.form = 0
        again = autotune.tune(dp, types.SimpleNamespace(precision=0))
        assert again["cached"] and again["best"] == (64, 2, 8, 4) and lib.form == 4, again
