"""The forward row DST of many layers and of several rows per CTA, with the
predictor (adaptive dt) and without: the mixed form against the oracle, and
the time of the predictor -- five more loads and two more stores of a layer's
node beside the projection's one load and the transform: at most 2.5 times
the time of the projection alone (spilled registers, or loads that wait for
one another, take it to 2.9 and 3.4)."""
import numpy as np
import pytest

import pequod_b200 as pq
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def gyre(ii, jj, L, precision, adapt):
    H = tuple(3.0e4 * (k + 1) for k in range(L))
    gp = tuple(1.5 * 2.0 ** -k for k in range(L - 1))
    return pq.Config.from_physical(pq.double_gyre_physical(ii, jj, layers=L, dt=900.0, dx=3.84e8 / (ii - 1), H=H,
                                                           gprime=gp, precision=precision, adapt_dt=adapt))


# Three steps, some ten FP32 roundings (6e-8) each, a factor of five between layers and modes.
TOL_MIXED = 1e-5


@pytest.mark.parametrize("adapt", [0, 1])
@pytest.mark.parametrize("ii,jj,L", [(5, 6, 6), (17, 9, 3), (17, 14, 7), (33, 10, 8), (65, 7, 5), (65, 9, 6), (129, 6, 8),
                                     (257, 5, 7), (513, 6, 6), (1025, 5, 6), (1025, 6, 8), (2049, 5, 6)])
def test_mixed_against_oracle(ii, jj, L, adapt):
    cfg = gyre(ii, jj, L, pq.PREC_MIXED, adapt)
    ic = pq.make_ic(ii, jj, L, seed=ii + jj, amplitude=1e-7 * cfg.t_scale, sigma=2.0)
    g, o = pq.Model(cfg), O.Model(O.cfg_from(cfg))
    g.init_perturb(ic)
    o.init(ic)
    g.step(3)
    o.step(3)
    a, b = g.sdata("psi"), o.get("psi")[1:-1, 1:-1]
    g.close()
    assert np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()) <= TOL_MIXED


LANES = [(5, 1), (9, 1), (9, 2), (17, 1), (17, 4), (33, 1), (33, 2), (129, 16)]


@pytest.mark.parametrize("ii,tune,precision", [(ii, dict(dst_lanes=p), prec) for ii, p in LANES
                                               for prec in (pq.PREC_FP64, pq.PREC_MIXED)]
                         + [(129, dict(dst_algo=2), pq.PREC_MIXED)])
def test_predictor_of_other_geometries(ii, tune, precision):
    """Seven layers, adaptive: pairs of fewer nodes than a warp has lanes among them."""
    cfg = gyre(ii, 11, 7, precision, 1)
    ic = pq.make_ic(ii, 11, 7, seed=ii, amplitude=1e-7 * cfg.t_scale, sigma=2.0)
    g, o = pq.Model(cfg), O.Model(O.cfg_from(cfg))
    g.set_tuning(**tune)
    g.init_perturb(ic)
    o.init(ic)
    g.step(3)
    o.step(3)
    a, b = g.sdata("psi"), o.get("psi")[1:-1, 1:-1]
    g.close()
    assert np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()) <= (1e-12 if precision == pq.PREC_FP64 else TOL_MIXED)


def forward_us(precision, adapt):
    cfg = gyre(1025, 257, 8, precision, adapt)
    m = pq.Model(cfg)
    m.init_perturb(pq.make_ic(1025, 257, 8, seed=1, amplitude=1e-8 * cfg.t_scale, sigma=2.0))
    m.step(2)
    best = 1e30
    for _ in range(5):
        m.kernel_timing(True)
        for _ in range(10):
            m.step_async(1)
        ms, n = m.kernel_times()["dst_forward"]
        m.kernel_timing(False)
        best = min(best, 1e3 * ms / n)
    m.close()
    return best


@pytest.mark.parametrize("precision", [pq.PREC_FP64, pq.PREC_MIXED])
def test_time_of_the_predictor(precision):
    assert forward_us(precision, 1) <= 2.5 * forward_us(precision, 0)
