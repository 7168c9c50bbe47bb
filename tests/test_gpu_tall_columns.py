"""Grids of more than 2050 rows, whose tridiagonal chunks do not fit registers:
the solve against the oracle's helm at the edges of its shared-memory split
(1e-12 as the other solves), and its time, which grows with the rows -- at
most twice what a row of the 2050-row grid costs (the strip in shared memory
holds fewer CTAs per SM; instances that spill cost 2.5 to 8 times as much)."""
import numpy as np
import pytest

import pequod_b200 as pq
from oracle import oracle as O
from pequod_b200.workloads import double_gyre

pytestmark = pytest.mark.gpu


def helm_cfg(ii, jj, ss, periodic):
    d = pq.ModelDesc()
    d.ii, d.jj, d.layers, d.periodic_j = ii, jj, len(ss), int(periodic)
    d.limiter, d.bc_type, d.dt = 1, pq.BC_FREE_SLIP, 1.0
    for k in range(len(ss)):
        d.ss[k], d.h[k] = ss[k], 1.0
        d.m2z[k + len(ss) * k] = d.z2m[k + len(ss) * k] = 1.0
    return pq.Config(d, None, 1.0)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("jj", [2051, 2114, 2115, 3601, 7105, 7106, 7107, 8193, 8194])
def test_helm_tall(jj, periodic):
    ss = [0.0, 1e-3, 0.3] if not periodic else [1e-3, 0.3]
    m = pq.Model(helm_cfg(9, jj, ss, periodic))
    z = np.asfortranarray(np.random.default_rng(jj).standard_normal((9, jj, len(ss))))
    a, b = m.helm(z), O.Helm(9, jj, len(ss), np.array(ss), periodic_j=periodic)(z)
    assert np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()) <= 1e-12
    m.close()


def test_taller_is_refused():
    with pytest.raises(pq.PQError):
        m = pq.Model(helm_cfg(9, 8195, [1e-3], False))
        m.helm(np.zeros((9, 8195, 1), order="F"))


def tridiag_us(jj, precision):
    cfg = double_gyre(257, 3, 900.0, precision, jj=jj)
    m = pq.Model(cfg)
    m.init_perturb(pq.make_ic(257, jj, 3, seed=1, amplitude=1e-8 * cfg.t_scale, sigma=2.0))
    m.step(2)
    best = 1e30
    for _ in range(5):
        m.kernel_timing(True)
        for _ in range(10):
            m.step_async(1)
        ms, n = m.kernel_times()["tridiag"]
        m.kernel_timing(False)
        best = min(best, 1e3 * ms / n)
    m.close()
    return best


@pytest.mark.parametrize("precision", [pq.PREC_FP64, pq.PREC_MIXED])
def test_time_grows_with_the_rows(precision):
    per_row = tridiag_us(2050, precision) / 2050
    slow = {jj: t for jj in (2600, 4500, 6000) if (t := tridiag_us(jj, precision)) > 2 * per_row * jj}
    assert slow == {}
