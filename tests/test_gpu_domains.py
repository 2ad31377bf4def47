"""Uneven regional domains stepped by one persistent kernel, through the C-ABI.

Every domain of a batch must come out exactly as if it had been stepped on its
own: bit-identical to the CPU oracle in FP64, bit-identical to the handle API
at the same precision in both FP64 and mixed form, whatever the launch shape,
with or without the CUDA graph. A domain whose input is never published makes
the step end with a timeout status (bounded waits), and the next step runs.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU-only container
    pytest.skip("needs a CUDA device", allow_module_level=True)

from more_benchmarks_dc_ocean_b200 import inputs  # noqa: E402
from oracle import oracle as O  # noqa: E402

# Odd extents (PPM offsets off any power of two), nz from 1 to 25, 6 tracers.
SHAPES = [(21, 17, 5), (33, 25, 9), (40, 31, 12), (16, 29, 25), (57, 19, 7), (12, 12, 3), (9, 40, 1), (30, 30, 16)]


def _domains():
    ps = [inputs.make_problem(a, b, c, n_seamounts=3, land_fraction=0.2, n_passive=4, seed=900 + d,
                              name=f"d{d}_{a}x{b}x{c}") for d, (a, b, c) in enumerate(SHAPES)]
    ps[3].walls = (0, 1, 0, 0)  # open west / south / north edges on one domain
    return ps


def _assert_exact(name, a, b):
    a, b = np.asarray(a), np.asarray(b)
    if not np.array_equal(a, b):
        d = np.abs(a - b)
        pytest.fail(f"{name}: {int(np.count_nonzero(a != b))} values differ, max |diff| {d.max():.3e}")


def _batch_run(R, ps, nsteps, precision=0, occupancy=0, account=False, **kw):
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps, precision=precision, **kw)
    if occupancy:
        b.set_tuning(b.tile, b.chunk, occupancy)
        assert b.get_tuning()["occupancy"] == occupancy
    if account:
        b.set_accounting(True)
    b.step(nsteps)
    torch.cuda.synchronize()
    st = b.status()
    if account:  # every tile of the last step is accounted for, once
        tiles = sum(v["tiles"] for v in b.stage_times().values())
        assert tiles == b.items, (tiles, b.items)
    b.destroy()
    assert st["status"] == 0 and st["bad"] == 0, st
    return [[t.cpu().numpy() for t in dp.ms.tracers] for dp in dps]


def _handle_run(R, p, nsteps, precision=0):
    dp = R.to_device(p)
    redi = R.make_redi(dp, precision)
    R.step(dp, redi, nsteps)
    torch.cuda.synchronize()
    assert redi.error_count() == 0
    redi.destroy()
    return [t.cpu().numpy() for t in dp.ms.tracers]


def test_batch_fp64_matches_oracle(redi_lib, oracle_lib):
    """Two steps of eight uneven domains in one launch each: every tracer equals the oracle's, 0 ulp."""
    ps = _domains()
    got = _batch_run(redi_lib, ps, 2)
    for p, g in zip(ps, got):
        q = p.copy()
        O.step(q, 2)
        for n, (a, b) in enumerate(zip(g, q.tracers)):
            _assert_exact(f"{p.name} tracer {n}", a, b)


@pytest.mark.parametrize("tile,chunk,graph,occ", [((32, 4), 8, False, 0), ((16, 8), 4, True, 5),
                                                  ((128, 1), 16, True, 6), ((8, 16), 8, True, 0)])
def test_batch_launch_shapes_identical(redi_lib, tile, chunk, graph, occ):
    """Results do not depend on the gather tile, the vertical chunk, the register budget or the graph."""
    ps = _domains()
    ref = _batch_run(redi_lib, ps, 1)
    got = _batch_run(redi_lib, ps, 1, occupancy=occ, account=True, tile=tile, chunk=chunk, use_graph=graph)
    for p, a, b in zip(ps, got, ref):
        for n in range(len(a)):
            _assert_exact(f"{p.name} tracer {n} tile {tile} chunk {chunk} graph {graph} occ {occ}", a[n], b[n])


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_matches_single_domain_handle(redi_lib, precision):
    """Per domain, the batch equals the handle API at the same precision (FP64 and mixed), bit for bit."""
    ps = _domains()[:5]
    got = _batch_run(redi_lib, ps, 2, precision=precision)
    for p, g in zip(ps, got):
        ref = _handle_run(redi_lib, p, 2, precision)
        for n, (a, b) in enumerate(zip(g, ref)):
            _assert_exact(f"{p.name} tracer {n} precision {precision}", a, b)


def test_batch_mixed_close_to_oracle(redi_lib, oracle_lib):
    """Mixed form after one step: relative error per domain at most 1e-7 of each tracer's scale."""
    ps = _domains()
    got = _batch_run(redi_lib, ps, 1, precision=1)
    for p, g in zip(ps, got):
        q = p.copy()
        O.step(q, 1)
        for n, (a, b) in enumerate(zip(g, q.tracers)):
            scale = max(float(np.abs(b).max()), 1e-300)
            err = float(np.abs(a - b).max()) / scale
            assert err <= 1e-7, f"{p.name} tracer {n}: {err:.3e}"


def test_batch_timeout_is_reported_and_recoverable(redi_lib):
    """A held domain's tiles give up after the wait limit; the status names it; the next step runs clean."""
    R = redi_lib
    ps = _domains()
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps)
    b.set_wait_limit(20_000_000)  # 20 ms
    b.hold(2)
    b.step()
    st = b.status()
    assert st["status"] == R.STATUS_TIMEOUT, st
    assert st["domain"] == 2 and st["stage"] in (0, 1), st
    b.hold(2, False)
    b.step()
    assert b.status()["status"] == 0
    b.destroy()


def test_batch_rejects_bad_arguments(redi_lib):
    R = redi_lib
    p = inputs.make_problem(12, 10, 4, seed=1)
    dp = R.to_device(p)
    with pytest.raises(R.RediError, match="128 cells"):
        R.RediBatch([dp], tile=(16, 4))
    with pytest.raises(R.RediError, match="chunk"):
        R.RediBatch([dp], chunk=5)
    dp1 = R.to_device(p, tracers=p.tracers[:1])
    dp1.ms.idx_salinity = 0
    with pytest.raises(R.RediError, match="tracers"):
        R.RediBatch([dp1])
    dp.khtr_u_ext = None
    with pytest.raises(R.RediError, match="NULL"):
        R.RediBatch([dp])


@pytest.mark.parametrize("precision,graph,swap", [(0, True, False), (0, False, True), (1, True, False)])
def test_batch_forms_identical(redi_lib, precision, graph, swap):
    """The persistent kernel and the launches per domain give the same bits over three steps, with T and S
    in either order, and a step may change form."""
    R = redi_lib
    ps = _domains()
    if swap:
        for p in ps[:2]:
            p.tracers[0], p.tracers[1] = p.tracers[1], p.tracers[0]
            p.idx_temperature, p.idx_salinity = p.idx_salinity, p.idx_temperature
        ps[2].tracers[1], ps[2].tracers[4] = ps[2].tracers[4], ps[2].tracers[1]
        ps[2].idx_salinity = 5
    out = []
    for forms in ((R.BATCH_PERSISTENT,) * 3, (R.BATCH_LAUNCHES, R.BATCH_PERSISTENT, R.BATCH_LAUNCHES)):
        dps = [R.to_device(p) for p in ps]
        b = R.RediBatch(dps, precision=precision, use_graph=graph)
        for f in forms:
            b.set_form(f)
            assert b.get_form() == f
            b.step()
            st = b.status()
            assert st["status"] == 0 and st["bad"] == 0, st
        torch.cuda.synchronize()
        b.destroy()
        out.append([[t.cpu().numpy() for t in dp.ms.tracers] for dp in dps])
    for p, x, y in zip(ps, out[1], out[0]):
        for n in range(len(x)):
            _assert_exact(f"{p.name} tracer {n}", x[n], y[n])


def test_batch_launches_time_out_on_a_held_domain(redi_lib):
    """The launches per domain: a held domain ends the step with the status, no tracer is touched, and the
    next step runs."""
    R = redi_lib
    ps = _domains()[:3]
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps)
    b.set_form(R.BATCH_LAUNCHES)
    b.set_wait_limit(20_000_000)  # 20 ms
    b.hold(1)
    b.step()
    st = b.status()
    assert st["status"] == R.STATUS_TIMEOUT and st["domain"] == 1 and st["stage"] == 0, st
    for p, dp in zip(ps, dps):
        for a, t in zip(p.tracers, dp.ms.tracers):
            _assert_exact(f"{p.name} untouched", t.cpu().numpy(), a)
    b.hold(1, False)
    b.step()
    assert b.status()["status"] == 0
    got = [[t.cpu().numpy() for t in dp.ms.tracers] for dp in dps]
    b.destroy()
    for p, g in zip(ps, got):
        ref = _handle_run(R, p, 1)
        for n, (a, c) in enumerate(zip(g, ref)):
            _assert_exact(f"{p.name} tracer {n}", a, c)


def test_batch_goes_on_around_a_held_domain(redi_lib):
    """Left to itself, a step with a held domain names it in the status and advances every other domain by
    one step; the held one is untouched, and a form that the caller chose stays in force."""
    R = redi_lib
    ps = _domains()
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps)
    assert b.get_form() == R.BATCH_LAUNCHES
    b.set_wait_limit(100_000_000)  # 100 ms: the other domains take a fraction of one
    b.hold(2)
    assert b.get_form() == R.BATCH_PERSISTENT
    b.step()
    st = b.status()
    assert st["status"] == R.STATUS_TIMEOUT and st["domain"] == 2 and st["stage"] in (0, 1), st
    for k, (p, dp) in enumerate(zip(ps, dps)):
        ref = p.tracers if k == 2 else _handle_run(R, p, 1)
        for n, (t, c) in enumerate(zip(dp.ms.tracers, ref)):
            _assert_exact(f"{p.name} tracer {n}", t.cpu().numpy(), c)
    b.hold(2, False)
    assert b.get_form() == R.BATCH_LAUNCHES
    b.step()
    assert b.status()["status"] == 0
    b.set_form(R.BATCH_LAUNCHES)
    b.hold(2)
    assert b.get_form() == R.BATCH_LAUNCHES
    b.destroy()


@pytest.mark.parametrize("n,shape,npas,launches", [(12, (16, 16, 8), 0, True), (200, (16, 16, 8), 0, False),
                                                   (200, (10, 9, 5), 3, False), (1, (6, 6, 1), 0, True)])
def test_batch_form_by_size(redi_lib, n, shape, npas, launches):
    """Left to itself, a batch of many small domains takes one kernel, others the launches; the step is the
    other form's bit for bit."""
    R = redi_lib
    ps = [inputs.make_problem(*shape, n_seamounts=3, land_fraction=0.2, n_passive=npas, seed=50 + k) for k in range(3)]
    out = []
    for form in (R.BATCH_AUTO, R.BATCH_PERSISTENT if launches else R.BATCH_LAUNCHES):
        dps = [R.to_device(ps[k % 3]) for k in range(n)]
        b = R.RediBatch(dps)
        b.set_form(form)
        assert (b.get_form() == R.BATCH_LAUNCHES) == (launches == (form == R.BATCH_AUTO))
        b.step(2)
        st = b.status()
        b.destroy()
        assert st["status"] == 0 and st["bad"] == 0, st
        out.append([[t.cpu().numpy() for t in dp.ms.tracers] for dp in dps])
    for k, (x, y) in enumerate(zip(*out)):
        for i, (a, c) in enumerate(zip(x, y)):
            _assert_exact(f"domain {k} tracer {i}", a, c)


@pytest.mark.parametrize("npas,eos,precision", [(0, 1, 0), (0, 2, 0), (1, 2, 1), (4, 1, 0), (6, 1, 1), (10, 2, 0)])
def test_batch_memory(redi_lib, npas, eos, precision):
    """A batch takes the bytes of the coefficients and of the phases one after the other (Phase A's state in
    the bytes of Phase B's buffers, fluxes of two tracers), with T and S alone less than a tenth more."""
    R = redi_lib
    small = R.to_device(inputs.make_problem(12, 10, 4, n_passive=npas, seed=3))
    b = R.RediBatch([small], precision=precision)  # the kernels are loaded
    b.step()
    b.destroy()
    p = inputs.make_problem(260, 180, 40, n_passive=npas, seed=3)
    dp = R.to_device(p)
    dp.eos.variant = eos
    nx, ny, nz, ntr = p.nx, p.ny, p.nz, p.ntr
    faces, ncol, ns = (nx + 1) * ny + nx * (ny + 1), nx * ny, 2 * nz + 2
    ko, f = (2, 4) if precision else (4, 8)
    coef = faces * (ns * (16 + 2 * ko) + (ns - 1) * f + 1)
    in_turn = max(40 * ncol * (nz + 1), ntr * ncol * (8 * (nz + 1) + 4 * f * nz) + 2 * (ns - 1) * faces * f)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    b = R.RediBatch([dp], precision=precision)
    used = free - torch.cuda.mem_get_info()[0]
    b.destroy()
    assert used <= (coef + in_turn) * (1.1 if npas == 0 else 1.0) + (8 << 20), (used, coef + in_turn)


@pytest.mark.parametrize("npas", [0, 1, 3, 7, 10])
@pytest.mark.parametrize("setting", ["default", "group 1", "group 8", "sweep 3", "sweep 0", "gather 4", "gather 8",
                                     "staged", "fold"])
def test_batch_launches_under_other_settings(redi_lib, npas, setting):
    """The launches per domain under every process-wide form, and with T and S in other places: the handle's
    bits (its own tests compare those with the oracle)."""
    from more_benchmarks_dc_ocean_b200 import autotune as T

    R = redi_lib
    ps = [inputs.make_problem(*s, n_seamounts=3, land_fraction=0.2, n_passive=npas, seed=70 + k)
          for k, s in enumerate([(21, 17, 5), (19, 26, 27), (33, 8, 1)])]
    ps[1].tracers[0], ps[1].tracers[1] = ps[1].tracers[1], ps[1].tracers[0]
    ps[1].idx_temperature, ps[1].idx_salinity = 1, 0
    if npas:
        ps[2].tracers[1], ps[2].tracers[2] = ps[2].tracers[2], ps[2].tracers[1]
        ps[2].idx_salinity = 2
    want = [_handle_run(R, p, 2) for p in ps]
    saved = (T.get_tracer_group(), T.get_sweep_form(), T.get_gather_tracers(), T.get_flux_staged(), T.get_fold(),
             T.get_tuning())
    try:
        {"default": lambda: None, "group 1": lambda: T.set_tracer_group(1), "group 8": lambda: T.set_tracer_group(8),
         "sweep 3": lambda: T.set_sweep_form(3), "sweep 0": lambda: T.set_sweep_form(0),
         "gather 4": lambda: (T.set_tracer_group(4), T.set_gather_tracers(4, 1)),
         "gather 8": lambda: (T.set_tracer_group(4), T.set_tuning(64, 2, 4), T.set_gather_tracers(8, 1)),
         "staged": lambda: T.set_flux_staged(1), "fold": lambda: T.set_fold(T.FOLD_FP64)}[setting]()
        dps = [R.to_device(p) for p in ps]
        b = R.RediBatch(dps)
        b.set_form(R.BATCH_LAUNCHES)
        b.step(2)
        st = b.status()
        b.destroy()
    finally:
        T.set_tracer_group(saved[0])
        T.set_sweep_form(saved[1])
        T.set_tuning(*saved[5])
        T.set_gather_tracers(*saved[2])
        T.set_flux_staged(saved[3])
        T.set_fold(*saved[4])
    assert st["status"] == 0 and st["bad"] == 0, st
    for p, dp, ref in zip(ps, dps, want):
        for n, (t, c) in enumerate(zip(dp.ms.tracers, ref)):
            _assert_exact(f"{setting} {p.name} tracer {n}", t.cpu().numpy(), c)


@pytest.mark.parametrize("graph", [True, False])
def test_batch_launch_counts(redi_lib, graph):
    """The launch counter tells the sweep with fluxes from the plain one, and a step made of launches (its
    gate, and every domain's under their own ids) from the persistent kernel."""
    import ctypes as C

    R = redi_lib
    L = R.lib()
    L.redi_b200_launch_count.restype = C.c_ulonglong
    L.redi_b200_launch_count.argtypes = [C.c_int]

    def counts(call):
        before = [L.redi_b200_launch_count(k) for k in range(L.redi_b200_kernel_count())]
        call()
        return {k: n for k in range(len(before)) if (n := L.redi_b200_launch_count(k) - before[k])}

    ps = [inputs.make_problem(21, 17, 5, seed=1), inputs.make_problem(16, 12, 7, seed=2)]
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps, use_graph=graph)
    b.set_form(R.BATCH_LAUNCHES)
    b.step()
    assert counts(b.step) == {20: 1, 17: 2, 18: 2, 3: 2}  # gate; columns, sweep with fluxes, gather of two domains
    b.set_form(R.BATCH_PERSISTENT)
    b.step()
    assert counts(b.step) == {8: 1}
    b.destroy()
    redi = R.make_redi(dps[0])
    assert counts(lambda: R.step(dps[0], redi, 1)) == {17: 1, 18: 1, 3: 1}
    torch.cuda.synchronize()
    redi.destroy()


@pytest.mark.parametrize("form", ["persistent", "launches"])
def test_batch_forms_match_oracle(redi_lib, oracle_lib, form):
    """Two steps of uneven domains with every equation of state, in either form: the oracle's bits."""
    R = redi_lib
    ps = _domains()
    for k, p in enumerate(ps):
        p.eos.variant = (1, 2, 4)[k % 3]
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps)
    b.set_form(R.BATCH_PERSISTENT if form == "persistent" else R.BATCH_LAUNCHES)
    b.step(2)
    st = b.status()
    b.destroy()
    assert st["status"] == 0 and st["bad"] == 0, st
    for p, dp in zip(ps, dps):
        q = p.copy()
        O.step(q, 2)
        for n, (t, c) in enumerate(zip(dp.ms.tracers, q.tracers)):
            _assert_exact(f"{p.name} eos {p.eos.variant} tracer {n}", t.cpu().numpy(), c)


@pytest.mark.parametrize("precision", [0, 1])
def test_persistent_kernel_times_out_and_recovers(redi_lib, precision):
    """The persistent kernel's bounded waits: the held domain is named, its tracers stay, and the next step
    runs from where the others are."""
    R = redi_lib
    ps = _domains()[:4]
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps, precision=precision)
    b.set_form(R.BATCH_PERSISTENT)
    b.set_wait_limit(100_000_000)  # 100 ms: the other domains take a fraction of one
    b.hold(3)
    b.step()
    st = b.status()
    assert st["status"] == R.STATUS_TIMEOUT and st["domain"] == 3 and st["stage"] in (0, 1), st
    b.hold(3, False)
    b.step()
    assert b.status()["status"] == 0
    b.destroy()
    for k, (p, dp) in enumerate(zip(ps, dps)):
        ref = _handle_run(R, p, 1 if k == 3 else 2, precision)
        for n, (t, c) in enumerate(zip(dp.ms.tracers, ref)):
            _assert_exact(f"{p.name} tracer {n}", t.cpu().numpy(), c)


def test_timeout_names_the_held_stage(redi_lib):
    """All stages of a small batch are claimed at almost the same time; the status names the held domain's
    column state every time, not a stage that waits behind it."""
    R = redi_lib
    ps = _domains()
    dps = [R.to_device(p) for p in ps]
    b = R.RediBatch(dps)
    b.set_form(R.BATCH_PERSISTENT)
    b.set_wait_limit(2_000_000)  # 2 ms
    for k in range(40):
        b.hold(k % len(ps))
        b.step()
        st = b.status()
        assert st["status"] == R.STATUS_TIMEOUT and st["domain"] == k % len(ps) and st["stage"] == 0, (k, st)
        b.hold(k % len(ps), False)
    b.step()
    assert b.status()["status"] == 0
    b.destroy()


def test_batch_fits_where_the_phases_in_turn_fit(redi_lib):
    """With room for a little more than the phases in turn, a batch of T and S alone is created without the
    bytes that its launches would take beyond them, and its step is the handle's."""
    R = redi_lib
    b = R.RediBatch([R.to_device(inputs.make_problem(12, 10, 4, seed=3))])  # the kernels are loaded
    b.step()
    b.destroy()
    p, n, mib = inputs.make_problem(200, 200, 25, seed=3), 30, 1 << 20
    dps = [R.to_device(p) for _ in range(n)]
    nx, ny, nz = p.nx, p.ny, p.nz
    faces, ncol, ns = (nx + 1) * ny + nx * (ny + 1), nx * ny, 2 * nz + 2
    coef = faces * (ns * 24 + (ns - 1) * 8 + 1)
    in_turn = 2 * ncol * (8 * (nz + 1) + 32 * nz) + 2 * (ns - 1) * faces * 8
    need = n * ((coef + in_turn) // (2 * mib) + 2) * 2 * mib + 64 * mib
    assert n * ncol * 16 * (nz + 1) > 256 * mib  # the state of both scalars beside the layers, less the interface values
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - need, dtype=torch.uint8, device="cuda")
    try:
        b = R.RediBatch(dps)
    finally:
        del filler
        torch.cuda.empty_cache()
    b.set_form(R.BATCH_LAUNCHES)
    b.step()
    assert b.status()["status"] == 0
    b.destroy()
    ref = _handle_run(R, p, 1)
    for k in (0, n // 2, n - 1):
        for i, (t, c) in enumerate(zip(dps[k].ms.tracers, ref)):
            _assert_exact(f"domain {k} tracer {i}", t.cpu().numpy(), c)
