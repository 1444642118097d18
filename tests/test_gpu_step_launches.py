"""A run's steps however they are launched: graphs, a graph of the rest, single
launches, the step's end in its last kernel or in a launch of its own.

sfg_advance(max_steps = k) for k around the graph length must give the bits,
the time and the step count of k sfg_step calls at its step sizes (which commit
every step with a launch of their own), and must do so again when the same run
is repeated (the second one replays a captured rest)."""
import numpy as np
import pytest

from sonicsolver_b200 import capi, cases


def _grid(name):
    if name == "tiles2d":
        return cases.isentropic_vortex(48, recipe="teno5Rusanov"), {}
    if name == "sweeps3d":
        return cases.taylor_green(16), {"variant": 0}
    if name == "tiles3d":
        return cases.taylor_green(16), {"variant": 1}
    if name == "curved":
        return cases.wavy_vortex(32, recipe="weno5Rusanov"), {}
    if name == "laws":
        c = cases.sod_1d(60)
        c.bc_lo, c.bc_hi = (capi.BC_LAW, 0, 0), (capi.BC_LAW, 0, 0)
        return c, {"variant": 1}
    if name == "cluster1d":
        return cases.sod_1d(90), {}
    return cases.sod_1d(90), {"variant": 1}


@pytest.mark.gpu
@pytest.mark.parametrize("time_recipe", ["SSPRK3", "forwardEuler", "classicalRK4"])
@pytest.mark.parametrize("precision", [capi.PREC_FP64, capi.PREC_FP32_FLUX])
@pytest.mark.parametrize("name", ["tiles1d", "tiles2d", "sweeps3d", "tiles3d", "curved", "laws"])
def test_advance_equals_single_steps(name, precision, time_recipe):
    case, kw = _grid(name)
    G = 4

    def solver():
        s = case.solver(precision=precision, time_recipe=time_recipe, cfl=0.2)
        if "variant" in kw:
            s.variant = kw["variant"]
        return s

    a, b = solver(), solver()
    q0 = np.ascontiguousarray(case.q)
    for k in (1, 3, 3, 3, G, G + 1, G + 1, 2 * G + 3):
        a.upload(q0)
        st, dts = a.advance(1e30, max_steps=k, graph_steps=G, dt_capacity=16)
        assert st.steps == k and len(dts) == k and st.last_dt == dts[-1]
        b.upload(q0)
        for dt in dts:
            b.step(float(dt))
        assert a.time() == b.time()
        np.testing.assert_array_equal(a.download(), b.download())
    # a run that ends on time: the same end however the graph's rest is launched
    t_end = 2.5 * dts[0] + dts[1]
    ends = []
    for g in (1, 3, 64):
        a.upload(q0)
        st, d = a.advance(t_end, graph_steps=g, dt_capacity=16)
        assert abs(st.time - t_end) <= 1e-14 * max(1.0, t_end)
        ends.append((st.steps, a.download()))
    for n, q in ends[1:]:
        assert n == ends[0][0]
        np.testing.assert_array_equal(q, ends[0][1])


@pytest.mark.gpu
@pytest.mark.parametrize("time_recipe", ["SSPRK3", "forwardEuler", "classicalRK4"])
@pytest.mark.parametrize("name", ["tiles1d", "cluster1d", "tiles2d", "sweeps3d", "tiles3d", "curved", "laws"])
def test_advance_without_a_step_keeps_the_state(name, time_recipe):
    """A run that takes no step (its end time is reached) leaves a state handed
    over after an earlier run as it is, to the bit."""
    case, kw = _grid(name)
    s = case.solver(time_recipe=time_recipe, cfl=0.2)
    if "variant" in kw:
        s.variant = kw["variant"]
    s.advance(1e30, max_steps=3, graph_steps=2)
    q = np.ascontiguousarray(case.q * 1.25)
    for t_end, g in ((3.0, 2), (2.0, 1)):
        s.upload(q, 3.0)
        before = s.download()
        st, _ = s.advance(t_end, graph_steps=g)
        assert st.steps == 0 and s.time() == (3.0, 0)
        np.testing.assert_array_equal(s.download(), before)


@pytest.mark.gpu
@pytest.mark.parametrize("time_recipe", ["SSPRK3", "forwardEuler", "classicalRK4"])
@pytest.mark.parametrize("name", ["tiles1d", "tiles2d", "sweeps3d", "tiles3d", "curved", "laws"])
def test_cfl_step_is_one_step_of_a_run(name, time_recipe):
    """sfg_step without a dt: the CFL step from the state handed over, at the
    run's dt, with its bits; a limit clips it; an invalid state is refused and
    stays as it is."""
    case, kw = _grid(name)
    a, b = (case.solver(time_recipe=time_recipe, cfl=0.2) for _ in range(2))
    for s in (a, b):
        if "variant" in kw:
            s.variant = kw["variant"]
    _, dts = a.advance(1e30, max_steps=3, dt_capacity=3)
    for k in range(3):
        b.step()
        assert b.time() == (float(sum(dts[:k + 1])), k + 1)
    np.testing.assert_array_equal(a.download(), b.download())
    t, n = b.time()
    b.step(limit=0.25 * float(dts[2]))
    assert b.time() == (t + 0.25 * float(dts[2]), n + 1)
    bad = np.ascontiguousarray(case.q).copy()
    bad[0, -5 if case.dim > 1 else 0, 20 % case.n[0], 4] = np.nan
    b.upload(bad)
    before = b.download()
    with pytest.raises(capi.SolverError) as e:
        b.step()
    assert e.value.code == capi.ERR_STATE and b.time() == (0.0, 0)
    np.testing.assert_array_equal(b.download(), before)


@pytest.mark.gpu
def test_stream_that_cannot_be_captured():
    """The legacy default stream: runs of any length go launch by launch, with the
    bits of a captured one, and leave no error behind."""
    case, _ = _grid("tiles2d")
    a, b = case.solver(), case.solver(stream=1)  # 1: cudaStreamLegacy
    for kw in (dict(max_steps=9, graph_steps=4), dict(max_steps=70), dict(max_steps=2), dict(max_steps=2)):
        (sa, da), (sb, db) = (s.advance(1e30, dt_capacity=70, **kw) for s in (a, b))
        assert sa.steps == sb.steps == kw["max_steps"] and a.time() == b.time()
        np.testing.assert_array_equal(da, db)
        np.testing.assert_array_equal(a.download(), b.download())
    case.solver().advance(1e30, max_steps=2)


@pytest.mark.gpu
def test_device_time_leaves_the_capture_out():
    """stats.device_ms of the run that captures its graph behind its first steps:
    the steps' time, not that of capturing and instantiating 512 steps (7 ms,
    against 0.2 for the two steps)."""
    case, _ = _grid("tiles2d")
    case.solver().advance(1e30, max_steps=2, graph_steps=512)  # kernels loaded
    s = case.solver()
    first, again = (s.advance(1e30, max_steps=2, graph_steps=512)[0].device_ms for _ in range(2))
    assert 0.0 < first < 1.0 and 0.0 < again < 1.0
