"""The row DSTs at the edges of their geometry: the smallest and largest
lengths, every values-per-lane count, layer counts on both sides of the
unrolled ones, rows that do not fill a CTA -- against the oracle.  Tolerances
are those of a step in FP64 (1e-12) and of the mixed form (1e-6)."""
import numpy as np
import pytest

import pequod_b200 as pq
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def gyre(ii, jj, L, precision=pq.PREC_FP64, **kw):
    H = tuple(3.0e4 * (k + 1) for k in range(L))
    gp = tuple(1.5 * 2.0 ** -k for k in range(L - 1))
    return pq.Config.from_physical(pq.double_gyre_physical(ii, jj, layers=L, dt=900.0, dx=3.84e8 / (ii - 1), H=H,
                                                           gprime=gp, precision=precision, **kw))


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


SHAPES = [(5, 5, 1), (9, 6, 2), (17, 7, 8), (33, 9, 6), (65, 6, 8), (129, 5, 3), (129, 8, 7), (257, 7, 4),
          (513, 6, 5), (1025, 5, 3), (1025, 6, 8), (2049, 6, 5), (2049, 5, 6)]


@pytest.mark.parametrize("ii,jj,L", SHAPES)
def test_inversion_and_steps(ii, jj, L):
    tol = 1e-12
    for adapt in (0, 1):  # the projection alone, and fused with the predictor
        cfg = gyre(ii, jj, L, adapt_dt=adapt)
        ic = pq.make_ic(ii, jj, L, seed=ii + jj, amplitude=1e-7 * cfg.t_scale, sigma=2.0)
        g, o = pq.Model(cfg), O.Model(O.cfg_from(cfg))
        zd = np.zeros((ii + 2, jj + 2, L), order="F")
        zd[1:-1, 1:-1] = ic
        assert rel_l2(g.pv_inversion(ic), o.pv_inversion(zd)[1:-1, 1:-1]) <= tol
        g.init_perturb(ic)
        o.init(ic)
        g.step(3)
        o.step(3)
        assert rel_l2(g.sdata("psi"), o.get("psi")[1:-1, 1:-1]) <= tol
        g.close()


@pytest.mark.parametrize("lanes", [8, 16, 32, 64])
def test_mixed_trajectory_of_other_lanes(lanes):
    """Other lanes per unit (run-time geometry) give the default's result to rounding of FP32."""
    cfg = gyre(513, 9, 3, pq.PREC_MIXED)
    ic = pq.make_ic(513, 9, 3, seed=3, amplitude=1e-7 * cfg.t_scale, sigma=2.0)
    psi = []
    for tune in ({}, dict(dst_lanes=lanes, dst_lanes_inv=lanes)):
        m = pq.Model(cfg)
        if tune:
            m.set_tuning(**tune)
        psi.append(m.pv_inversion(ic))
        m.close()
    assert rel_l2(psi[1], psi[0]) <= 1e-6
