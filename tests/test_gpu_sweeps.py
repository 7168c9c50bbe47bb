"""The CABARET sweeps at the edges of their decomposition -- grids narrower
than a strip, bands taller than the grid or that leave a remainder, no or one
interior sweep, every layer position -- against the oracle (FP64, 1e-12 per
step as the other step tests) and, in the mixed form, against the tile
kernel's step (FP32 rounding of one step, 1e-6)."""
import numpy as np
import pytest

import pequod_b200 as pq
from oracle import oracle as O
from pequod_b200.workloads import double_gyre

pytestmark = pytest.mark.gpu

FIELDS = ["psi", "zeta", "ui", "uj", "zeta_fi", "zeta_fj", "res", "res_beta"]


def rel_l2(a, b):
    nb = np.linalg.norm(b.ravel())
    return float(np.linalg.norm((a - b).ravel()) / (nb if nb > 0 else 1.0))


def owned(a):
    return a[1:-1, 1:-1] if a.shape[0] % 2 else a


SHAPES = [(9, 9, 2, 4), (17, 40, 3, 128), (33, 11, 1, 5), (65, 21, 5, 7), (65, 64, 3, 4), (129, 33, 4, 9),
          (129, 50, 3, 17), (257, 29, 2, 6)]


@pytest.mark.parametrize("adapt", [0, 1])
@pytest.mark.parametrize("ii,jj,L,band", SHAPES)
def test_sweeps_against_oracle(ii, jj, L, band, adapt):
    cfg = double_gyre(ii, L, 900.0, jj=jj, adapt_dt=adapt)
    g, o = pq.Model(cfg), O.Model(O.cfg_from(cfg))
    g.set_tuning(cab_kernel=1, cab_band=band)
    ic = pq.make_ic(ii, jj, L, seed=ii * jj, amplitude=1e-7 * cfg.t_scale, sigma=2.0)
    g.init_perturb(ic)
    o.init(ic)
    for _ in range(3):
        g.step(1)
        o.step(1)
        assert {f: e for f in FIELDS if (e := rel_l2(owned(g.get(f)), owned(o.get(f)))) > 1e-12} == {}
        assert abs(g.cfl() - o.cfl()) <= 1e-12 * o.cfl()
    g.close()


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("ii,jj,L,band", SHAPES)
def test_mixed_sweeps_against_tiles(ii, jj, L, band, kernel):
    psi = []
    for k in (0, kernel):
        cfg = double_gyre(ii, L, 900.0, pq.PREC_MIXED, jj=jj)
        m = pq.Model(cfg)
        m.set_tuning(cab_kernel=k, cab_band=band)
        m.init_perturb(pq.make_ic(ii, jj, L, seed=ii * jj, amplitude=1e-7 * cfg.t_scale, sigma=2.0))
        m.step(3)
        psi.append(m.sdata("psi"))
        m.close()
    assert rel_l2(psi[1], psi[0]) <= 1e-6
