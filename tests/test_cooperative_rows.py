"""Result rows of the solver in which a warp solves one problem: its lanes share
the rows, and the solver adds the transverse velocities onto a row that it has
written before.  A component across the face normal passes through a solve
unchanged -- the star states keep their own side's, the sampled state takes one
side's -- so every row can be checked exactly; the same problems by one thread
each give the same bits."""
import numpy as np
import pytest

from m2c_gb300 import abi, warmstart

pytestmark = pytest.mark.gpu


def _problems(n, seed):
    rng = np.random.default_rng(seed)
    ids = rng.integers(0, 3, (2, n)).astype(np.int32)
    V = np.zeros((2, n, 5))
    V[:, :, 0] = np.choose(ids, [1000.0, 1.2, 1000.0]) * 10.0 ** rng.uniform(-0.15, 0.15, (2, n))
    V[:, :, 1:4] = rng.uniform(-60.0, 60.0, (2, n, 3))
    V[:, :, 4] = np.choose(ids, [1.0e7, 1.0e6, 1.0e7]) * 10.0 ** rng.uniform(-1.0, 1.5, (2, n))
    axis = rng.integers(0, 3, n)
    return V[0], ids[0].copy(), V[1], ids[1].copy(), np.eye(3)[axis], axis


@pytest.mark.parametrize("n", [1, 31, 1216])
def test_transverse_velocities_of_every_row(n):
    from m2c_gb300.solver import Solver
    cfg = warmstart.solver_config()
    cfg.n_materials = 3
    abi.set_material(cfg.mat[0], abi.EOS_SG, gamma=6.12, pc=3.43e8)
    abi.set_material(cfg.mat[1], abi.EOS_SG, gamma=1.4, pc=0.0)
    abi.set_material(cfg.mat[2], abi.EOS_NASG, gamma=1.19, pc=6.2e8, b=6.61e-4, q=0.0)
    s = Solver(cfg)
    for seed in range(8):
        *p, axis = _problems(n, 100 + seed)
        r = s.riemann_batch(*p)
        assert np.all(r["err"] == 0)
        for k in range(3):
            t = axis != k
            np.testing.assert_array_equal(r["Vsm"][t, 1 + k], p[0][t, 1 + k])
            np.testing.assert_array_equal(r["Vsp"][t, 1 + k], p[2][t, 1 + k])
            assert np.all((r["Vs"][t, 1 + k] == p[0][t, 1 + k]) | (r["Vs"][t, 1 + k] == p[2][t, 1 + k]))
    rep = -(-1300 // n)
    many = s.riemann_batch(*[np.concatenate([a] * rep) for a in p])   # more problems than warps
    for k in ("Vs", "id", "Vsm", "Vsp", "iters", "err"):
        np.testing.assert_array_equal(r[k], many[k][:n], err_msg=k)
        np.testing.assert_array_equal(r[k], many[k][-n:], err_msg=k)
    s.close()
