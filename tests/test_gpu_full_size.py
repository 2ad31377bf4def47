"""GPU parity at the benchmark configurations themselves, not only at reduced sizes.

* config 1, 1440x1080x75 (T, S): one FP64 step through the handle API and through the
  reference-compatible `redi_opt_launch` export; every coefficient and both tracers equal
  the CPU oracle's at 0 ulp.
* config 3, 720x576x50 (T, S and 32 passive tracers): one FP64 step at 0 ulp; the mixed
  form after one step within 1e-7 of each field's scale.
* config 4: the three largest of the 64 uneven regional domains, stepped together by the
  persistent kernel in FP64, each equal to the oracle at 0 ulp.

The oracle needs a few seconds per config-1 step on the host's cores. Host arrays are
compared one at a time to keep host memory within ~25 GB.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from more_benchmarks_dc_ocean_b200 import inputs  # noqa: E402
from oracle import oracle as O  # noqa: E402

COEFFS = ("uPoL", "uPoR", "uKoL", "uKoR", "uhEff", "vPoL", "vPoR", "vKoL", "vKoR", "vhEff")


def _exact(name, got, ref):
    got = np.asarray(got)
    if got.shape != ref.shape or not np.array_equal(got, ref):
        n = int(np.count_nonzero(got != ref)) if got.shape == ref.shape else -1
        pytest.fail(f"{name}: {n} values differ from the oracle (bar 0 ulp)")


@pytest.fixture(scope="module")
def config1_oracle(oracle_lib):
    p = inputs.config1()
    q = p.copy()
    c = O.step(q, 1)
    return p, c, q.tracers


def test_config1_handle_api_matches_oracle(redi_lib, config1_oracle):
    R = redi_lib
    p, co, to = config1_oracle
    dp = R.to_device(p)
    redi = R.make_redi(dp)
    assert R.redi_calc_coeffs(dp.grid, dp.metrics, dp.eos, redi, dp.ms) == R.OK
    assert R.redi_apply_flux(dp.grid, dp.metrics, redi, dp.ms, dp.dt, dp.khtr_u_ext, dp.khtr_v_ext, dp.bc) == R.OK
    torch.cuda.synchronize()
    assert redi.error_count() == 0
    cg = redi.coeffs()
    for k in COEFFS:
        _exact(f"config1 {k}", cg[k].cpu().numpy(), co[k])
    for n in range(2):
        _exact(f"config1 tracer {n}", dp.ms.tracers[n].cpu().numpy(), to[n])
    redi.destroy()
    del dp
    torch.cuda.empty_cache()


def test_config1_opt_launch_export_matches_oracle(redi_lib, config1_oracle):
    R = redi_lib
    p, co, to = config1_oracle
    dp = R.to_device(p)
    # slots as ocean_redi_init leaves them (Po = 0, Ko = 1, hEff = 0): the edge faces are never written
    out = {k: (torch.ones if "Ko" in k else torch.zeros)(co[k].shape, dtype=torch.int32 if "Ko" in k else torch.float64,
                                                        device="cuda") for k in COEFFS}
    ku, kv = torch.zeros_like(dp.khtr_u_ext), torch.zeros_like(dp.khtr_v_ext)
    m = dp.metrics
    R.redi_opt_launch(p.nx, p.ny, p.nz, p.dt, p.nghost, p.nx_phys, p.ny_phys, p.walls, dp.eos, dp.ms.h_layer,
                      dp.ms.tracers[0], dp.ms.tracers[1], m.wet_u, m.wet_v, out, dp.khtr_u_ext, dp.khtr_v_ext,
                      ku, kv, m.dy_cu, m.dx_cv, m.idxCu, m.idyCv, m.areaT)
    torch.cuda.synchronize()
    for k in COEFFS:
        _exact(f"redi_opt_launch {k}", out[k].cpu().numpy(), co[k])
    for n in range(2):
        _exact(f"redi_opt_launch tracer {n}", dp.ms.tracers[n].cpu().numpy(), to[n])
    del dp, out
    torch.cuda.empty_cache()


def test_config3_fp64_and_mixed(redi_lib, oracle_lib):
    from more_benchmarks_dc_ocean_b200 import precision_report as PR

    R = redi_lib
    p = inputs.config3()
    q = p.copy()
    O.step(q, 1)
    dp = R.to_device(p)
    redi = R.make_redi(dp)
    R.step(dp, redi, 1)
    torch.cuda.synchronize()
    assert redi.error_count() == 0
    redi.destroy()
    for n in range(p.ntr):
        _exact(f"config3 FP64 tracer {n}", dp.ms.tracers[n].cpu().numpy(), q.tracers[n])
    del dp
    dm = R.to_device(p)
    redi = R.make_redi(dm, R.MIXED)
    R.step(dm, redi, 1)
    torch.cuda.synchronize()
    redi.destroy()
    for n in range(p.ntr):
        got = dm.ms.tracers[n].cpu().numpy()
        if n < 2:
            c = PR.compare(got, q.tracers[n])
            assert c["max_rel"] <= 1e-7, (n, c)
        else:  # passive tracers cross zero: against the field's scale
            assert np.abs(got - q.tracers[n]).max() <= 1e-7 * np.abs(q.tracers[n]).max(), n
    del dm
    torch.cuda.empty_cache()


def test_config4_largest_domains_match_oracle(redi_lib, oracle_lib):
    R = redi_lib
    shapes = inputs.config4_shapes()
    order = sorted(range(len(shapes)), key=lambda d: -shapes[d][0] * shapes[d][1] * shapes[d][2])[:3]
    ps = [inputs.config4_domain(20261203, d, shapes[d]) for d in order]
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps, precision=R.FP64)
    b.step(1)
    torch.cuda.synchronize()
    st = b.status()
    b.destroy()
    assert st["status"] == 0 and st["bad"] == 0, st
    for p, dp in zip(ps, dps):
        q = p.copy()
        O.step(q, 1)
        for n in range(p.ntr):
            _exact(f"config4 {p.name} tracer {n}", dp.ms.tracers[n].cpu().numpy(), q.tracers[n])


def test_largest_domains_in_the_persistent_kernel(redi_lib):
    """The same domains in the batch's other form: the launches' bits (which the oracle's test compares)."""
    R = redi_lib
    shapes = inputs.config4_shapes()
    order = sorted(range(len(shapes)), key=lambda d: -shapes[d][0] * shapes[d][1] * shapes[d][2])[:3]
    ps = [inputs.config4_domain(20261203, d, shapes[d]) for d in order]
    out = []
    for form in (R.BATCH_LAUNCHES, R.BATCH_PERSISTENT):
        dps = [R.to_device(p) for p in ps]
        b = R.RediBatch(dps)
        b.set_form(form)
        b.step(1)
        st = b.status()
        b.destroy()
        assert st["status"] == 0 and st["bad"] == 0, st
        out.append([[t.cpu().numpy() for t in dp.ms.tracers] for dp in dps])
    for p, x, y in zip(ps, *out):
        for n in range(p.ntr):
            _exact(f"{p.name} tracer {n}", y[n], x[n])
