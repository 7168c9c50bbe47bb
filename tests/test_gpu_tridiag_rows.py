"""The tridiagonal solves at the edges of their row split -- one row, the last
and first lengths of every chunk size and warp count, remainders, columns
longer than the registers hold -- against the oracle's helm (1e-12), closed
and periodic; and a step (mass correction) at a few of them."""
import numpy as np
import pytest

import pequod_b200 as pq
from oracle import oracle as O
from pequod_b200.workloads import double_gyre

pytestmark = pytest.mark.gpu

ROWS = [5, 6, 9, 10, 11, 17, 33, 34, 35, 65, 66, 67, 130, 131, 258, 259, 306, 307, 386, 387, 450, 514, 515, 642, 770,
        1026, 1027, 1282, 2050, 2051, 4098, 4099, 5000]


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def helm_cfg(ii, jj, ss, periodic):
    d = pq.ModelDesc()
    d.ii, d.jj, d.layers, d.periodic_j = ii, jj, len(ss), int(periodic)
    d.limiter, d.bc_type, d.dt = 1, pq.BC_FREE_SLIP, 1.0
    for k in range(len(ss)):
        d.ss[k], d.h[k] = ss[k], 1.0
        d.m2z[k + len(ss) * k] = d.z2m[k + len(ss) * k] = 1.0
    return pq.Config(d, None, 1.0)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("jj", ROWS)
def test_helm_rows(jj, periodic):
    ss = [1e-3, 0.3]
    m = pq.Model(helm_cfg(17, jj, ss, periodic))
    z = np.asfortranarray(np.random.default_rng(jj).standard_normal((17, jj, 2)))
    assert rel_l2(m.helm(z), O.Helm(17, jj, 2, np.array(ss), periodic_j=periodic)(z)) <= 1e-12
    m.close()


@pytest.mark.parametrize("jj", [6, 35, 131, 307, 515, 1027])
def test_step_rows(jj):
    cfg = double_gyre(33, 3, 900.0, jj=jj)
    g, o = pq.Model(cfg), O.Model(O.cfg_from(cfg))
    ic = pq.make_ic(33, jj, 3, seed=jj, amplitude=1e-7 * cfg.t_scale, sigma=2.0)
    g.init_perturb(ic)
    o.init(ic)
    g.step(2)
    o.step(2)
    assert rel_l2(g.sdata("psi"), o.get("psi")[1:-1, 1:-1]) <= 1e-12
    g.close()
