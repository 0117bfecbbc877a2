"""The schedule of a Runge-Kutta stage changes no result.

Reconstruction and fluxes run beside the first Riemann pass or after it,
whichever a device flag of the stage before says (did it leave unfinished
solves), and the first pass hands a solve over after a budget of evaluations.
Each test compares the same step under several of these schedules to the bit,
and with the oracle: the flag goes 0 -> 1 -> 0 by uploads of a state whose
solves outlast a budget of 3 evaluations and of one without an interface.

Bound against the oracle: a solve stops within 1e-10 of the pressure scale
(1e5 Pa); where rounding moves the stopping iteration, a CFL step of
0.4 / 1500 s/m turns that into 3e-10 of the largest velocity in the gas
(1.2 kg/m3).  1e-8, the bound of the multi-step comparisons, covers it; stale
fluxes are an error of order one."""
import numpy as np
import pytest

from m2c_gb300 import abi, problems
from m2c_gb300.ensemble import Ensemble
from m2c_gb300.solver import FluidState, Solver
from oracle import binding as ob
from oracle import parity

pytestmark = pytest.mark.gpu
LIMIT = "M2CG_RIEMANN_EVAL_LIMIT"
COUNTS = ("interface_faces", "riemann_solves", "riemann_iterations", "riemann_errors", "clipped_faces",
          "clipped_cells", "nonphysical", "swept_cells")
INTEGRATORS = [abi.TS_FORWARD_EULER, abi.TS_RK2, abi.TS_RK3]


def _states(ts, mp_recon=abi.MPREC_CONSTANT, n=16):
    """(config, stirred two-material state, state without an interface); water
    below 995 kg/m3 is clipped, so that the counters move in every stage."""
    cfg, V, ID, phi = problems.shock_bubble(n=n, radius=0.25)
    cfg.ts_type, cfg.mp_recon = ts, mp_recon
    cfg.mat[0].rhomin = 995.0
    rng = np.random.default_rng(23)
    V[:, 1:4] += rng.uniform(-5.0, 5.0, (len(V), 3))
    V[:, 4] *= 10.0 ** rng.uniform(-0.2, 0.2, len(V))
    W = V.copy()
    W[:, 0] = 1000.0 * (1.0 + 0.01 * problems.uniform_noise(len(V), 5))
    return cfg, FluidState(V, ID, phi), FluidState(W, np.zeros_like(ID), np.abs(phi) + 1.0)


def _step(s, st, how, dt):
    """Uploads st, takes one step; the state and the counters' increments."""
    s.set_state(st)
    before = s.counters()
    if how == "run":
        s.run(1)
    else:
        s.AdvanceOneTimeStep(dt)
    after = s.counters()
    return s.get_state(), {k: after[k] - before[k] for k in COUNTS}


def _same(a, b, what):
    for x, y in ((a.V, b.V), (a.ID, b.ID), (a.Phi, b.Phi)):
        np.testing.assert_array_equal(x, y, err_msg=str(what))


@pytest.mark.parametrize("how", ["run", "advance"])
@pytest.mark.parametrize("mp_recon", [abi.MPREC_CONSTANT, abi.MPREC_LINEAR])
@pytest.mark.parametrize("ts", INTEGRATORS)
def test_unfinished_solves_of_one_step_do_not_reach_the_next(monkeypatch, ts, mp_recon, how):
    monkeypatch.setenv(LIMIT, "3")
    cfg, stirred, calm = _states(ts, mp_recon)
    want, dts = {}, {}
    for name, st in (("stirred", stirred), ("calm", calm)):
        s = Solver(cfg, st)
        dts[name] = s.ComputeTimeStepSize()[0]
        want[name] = _step(s, st, how, dts[name])
        s.close()
        o = ob.OracleSim(cfg)
        o.upload(st.V, st.ID, st.Phi)
        o.advance(dts[name])
        V, ID, phi = o.download()
        assert np.all(parity.velocity_normalized(want[name][0].V, V) < 1e-8), name
        assert parity.rel_linf(want[name][0].Phi, phi) < 1e-8
        np.testing.assert_array_equal(want[name][0].ID, ID)
    c = want["stirred"][1]
    assert c["riemann_iterations"] > 3 * c["riemann_solves"] > 0   # some solves outlast the budget
    assert want["calm"][1]["interface_faces"] == 0
    assert min(want[k][1]["clipped_faces"] for k in want) > 0
    s = Solver(cfg)
    for name in ("stirred", "calm", "calm", "stirred", "stirred", "calm", "stirred"):
        got, counts = _step(s, stirred if name == "stirred" else calm, how, dts[name])
        _same(got, want[name][0], name)
        assert counts == want[name][1], name
    s.close()


@pytest.mark.parametrize("mp_recon", [abi.MPREC_CONSTANT, abi.MPREC_LINEAR])
@pytest.mark.parametrize("ts", INTEGRATORS)
def test_evaluation_budget_changes_no_step(monkeypatch, ts, mp_recon):
    """No hand-over at all (budget 0: the flag stays 0), some and nearly every
    solve handed over; the residual call's order of the same kernels as well."""
    cfg, stirred, _ = _states(ts, mp_recon)
    ref = None
    for limit in ("0", "3", "6", "24"):
        monkeypatch.setenv(LIMIT, limit)
        s = Solver(cfg, stirred)
        R = s.ComputeResidual()
        s.run(2)
        s.run(4)
        got = s.get_state(), s.counters(), R
        s.close()
        if ref is None:
            ref = got
            continue
        _same(got[0], ref[0], limit)
        for k in COUNTS:
            assert got[1][k] == ref[1][k], (limit, k)
        np.testing.assert_array_equal(got[2], ref[2], err_msg=limit)


@pytest.mark.parametrize("sms,lanes", [(1, 1), (2, 1), (40, 1), (1, 8), (152, 4)])
def test_layout_of_the_second_pass_changes_no_step(monkeypatch, sms, lanes):
    """About 300 handed-over solves a stage: several a warp in one and in more
    rounds (8 and 16 warps), one a warp on all eight warps of a block (320
    warps), packed by the lane setting; the default has one a warp on four."""
    monkeypatch.setenv(LIMIT, "3")
    cfg, stirred, _ = _states(abi.TS_RK2)
    ref = None
    for env in ({}, {"M2CG_RIEMANN_STRAGGLER_SMS": str(sms), "M2CG_RIEMANN_STRAGGLER_LANES": str(lanes)}):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        s = Solver(cfg, stirred)
        s.run(3)
        got = s.get_state(), s.counters()
        s.close()
        if ref is None:
            ref = got
    _same(got[0], ref[0], (sms, lanes))
    for k in COUNTS:
        assert got[1][k] == ref[1][k], k


@pytest.mark.parametrize("ts", [abi.TS_RK2, abi.TS_RK3])
def test_ensemble_steps_do_not_depend_on_the_step_before(monkeypatch, ts):
    monkeypatch.setenv(LIMIT, "3")
    cfg, stirred, calm = _states(ts)
    states = {"stirred": (stirred, calm), "calm": (calm, calm)}

    def step(e, name):
        for i, st in enumerate(states[name]):
            e.member(i).set_state(st)
        before = [e.member(i).counters() for i in range(2)]
        e.run(1)
        after = [e.member(i).counters() for i in range(2)]
        return [e.member(i).get_state() for i in range(2)], [{k: a[k] - b[k] for k in COUNTS} for a, b in zip(after, before)]

    want = {}
    for name in states:
        e = Ensemble([cfg, cfg])
        want[name] = step(e, name)
        e.close()
    e = Ensemble([cfg, cfg])
    for name in ("stirred", "calm", "calm", "stirred", "stirred", "calm"):
        got, counts = step(e, name)
        for a, b in zip(got, want[name][0]):
            _same(a, b, name)
        assert counts == want[name][1], name
    e.close()


@pytest.mark.parametrize("batched", [False, True])
def test_steps_without_unfinished_solves_wait_for_nobody(monkeypatch, batched):
    """The second pass's head start holds a stage back only where the stage
    before left unfinished solves: ten calm steps of two stages under one of
    1e8 cycles (about 50 ms; the first step after an upload may hold) end
    within a quarter of the 1 s that twenty such waits take."""
    import time
    monkeypatch.setenv("M2CG_RIEMANN_HOLD_CYCLES", "100000000")
    cfg, _, calm = _states(abi.TS_RK2)
    e = Ensemble([cfg, cfg]) if batched else None
    members = [e.member(i) for i in range(2)] if batched else [Solver(cfg)]
    for m in members:
        m.set_state(calm)
    run = e.run if batched else members[0].run
    run(1)   # captures the step
    t0 = time.perf_counter()
    run(10)
    assert time.perf_counter() - t0 < 0.25
    (e or members[0]).close()
