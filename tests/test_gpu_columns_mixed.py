"""Every chunk length of the tridiagonal solves in the mixed form (FP32 rows)
against the oracle, full chunks and a remainder of each; the same chunk lengths
in launches that hold several runs (descriptors from the device array) equal
the runs alone; and the formulation a default context takes."""
import numpy as np
import pytest

import pequod_b200 as pq
from oracle import oracle as O
from pequod_b200.workloads import double_gyre

pytestmark = pytest.mark.gpu

# Rows per chunk of the instances: 2 (32 chunks), 3 .. 32 (64 chunks), strips.
ROWS = [7, 34, 50, 66, 67, 130, 160, 194, 258, 300, 386, 450, 514, 600, 770, 800, 1026, 1100, 1282, 1400, 1538, 1800, 2050,
        2051, 2500, 3600]

# One inversion: 2 log2(32) butterfly stages, two spectral stores and the psi
# they give, each 6e-8 of the FP32 modes, a factor of five between layers and modes.
TOL = 5e-6


def rel_l2(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("jj", ROWS)
def test_inversion_of_fp32_rows(jj):
    cfg = double_gyre(33, 3, 900.0, pq.PREC_MIXED, jj=jj)
    g, o = pq.Model(cfg), O.Model(O.cfg_from(cfg))
    z = np.asfortranarray(np.random.default_rng(jj).standard_normal((33, jj, 3)) * 1e-7 * cfg.t_scale)
    zd = np.zeros((35, jj + 2, 3), order="F")
    zd[1:-1, 1:-1] = z
    assert rel_l2(g.pv_inversion(z), o.pv_inversion(zd)[1:-1, 1:-1]) <= TOL
    g.close()


@pytest.mark.parametrize("precision", [pq.PREC_FP64, pq.PREC_MIXED])
@pytest.mark.parametrize("jj", [34, 50, 130, 160, 258, 300, 386, 450, 514, 600, 770, 800, 1026, 1100, 1282, 1400, 1538, 1800,
                                2050, 2051])
def test_merged_equal_alone(jj, precision):
    cfg = double_gyre(17, 2, 900.0, precision, jj=jj)
    ics = [pq.make_ic(17, jj, 2, seed=60 + k, amplitude=1e-7 * cfg.t_scale, sigma=2.0) for k in range(2)]
    srv = pq.Server(4 << 30)
    ids = [srv.submit(cfg, ic, 3) for ic in ics]
    srv.run_until_done(max_steps=3)
    for rid, ic in zip(ids, ics):
        m = pq.Model(cfg)
        m.init_perturb(ic)
        m.step(3)
        assert np.array_equal(srv.collect(rid)[0], m.get("psi")[1:-1, 1:-1, :])
        m.close()
    srv.close()


@pytest.mark.parametrize("ii,jj,L,precision,kernel", [
    (129, 129, 3, pq.PREC_FP64, 0), (513, 240, 3, pq.PREC_FP64, 0), (513, 241, 3, pq.PREC_FP64, 1), (65, 2000, 3, pq.PREC_FP64, 1),
    (513, 181, 3, pq.PREC_MIXED, 0), (513, 182, 3, pq.PREC_MIXED, 1), (257, 1500, 2, pq.PREC_MIXED, 1),
    (257, 1501, 2, pq.PREC_MIXED, 2), (9, 1501, 1, pq.PREC_MIXED, 2)])
def test_default_formulation(ii, jj, L, precision, kernel):
    """Tiles below 370000 cell-layers (280000 mixed), sweeps from there, two columns
    per lane above 1500 rows of the mixed form; bands of 4 to 40 rows, 24 for two columns."""
    cfg = double_gyre(ii, L, 900.0, precision, jj=jj)
    m = pq.Model(cfg)
    t = m.get_tuning()
    m.close()
    assert t["cab_kernel"] == kernel
    assert t["cab_band"] == 24 if kernel == 2 else 4 <= t["cab_band"] <= 40
