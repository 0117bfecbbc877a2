"""Rarefactions that end at p = -p_inf: there c^2 = 0, every fixed-step
Runge-Kutta step from the last state has a stage of density -infinity and
fails, and the integration halves its step until its step limit.  Two such
pairs (a Noble-Abel and a stiffened gas), with the iteration limits lowered so
that a solve takes seconds no longer: by one warp and by one thread each to the
same bits, and the failure and the star pressure of the oracle (the retry that
gives them calls no library function: its operations are the oracle's)."""
import ctypes as C

import numpy as np
import pytest

from m2c_gb300 import abi, warmstart

W = np.array([[556.3624244348359, 73.95278249332932, 10827.65571515472,
               1331.8565863166425, 469.6907362088376, 574313.1756040176],
              [32.487719200170396, -250.6902927552953, 501999.11480208684,
               1176.069354879554, 127.75489108686133, 2708879.2401365037]])
E = np.array([[1.0, 2.7715821888644427, 281722226.10533595, 0.00036383088115026483, 0.0,
               0.0, 2.762235547744144, 36555669.662353106, 0.0, 0.0],
              [1.0, 3.1810824183844724, 449594125.31414676, 0.0002733689429908276, 0.0,
               0.0, 4.87410423906204, 26755798.927757367, 0.0, 0.0]])


def _config(tol=1e-10, make=warmstart.solver_config):
    c = make(tol)
    c.maxits_main = c.maxits_bracket = 12
    return c


def _oracle():
    from oracle import binding as ob
    lib = ob.lib()
    out, it, err = np.zeros((2, 4)), np.zeros(2, np.int32), np.zeros(2, np.int32)
    cfg = _config()
    lib.orc_riemann_batch_eos(C.byref(cfg), C.c_int64(2), abi.dptr(W), abi.dptr(E), None, abi.dptr(out), abi.iptr(it),
                              abi.iptr(err))
    return out, it, err


def test_the_pairs_fail_at_the_vacuum_in_the_oracle():
    out, it, err = _oracle()
    assert np.all(err == 1) and np.all(it > 12)
    np.testing.assert_allclose(out[:, 0], -E[:, 7], rtol=1e-3)   # next to the vacuum


@pytest.mark.gpu
def test_steps_to_the_vacuum(monkeypatch):
    monkeypatch.setattr(warmstart, "solver_config", _config)
    b = warmstart.BatchSolver()
    few = b.solve(W, E)
    many = b.solve(np.tile(W, (700, 1)), np.tile(E, (700, 1)))   # more problems than warps
    for k in ("pstar", "ustar", "rhol", "rhor", "iters", "err"):
        np.testing.assert_array_equal(np.tile(few[k], 700), many[k], err_msg=k)
    out, it, err = _oracle()
    np.testing.assert_array_equal(few["err"], err)
    np.testing.assert_allclose(few["pstar"], out[:, 0], rtol=1e-12)
    b.close()
