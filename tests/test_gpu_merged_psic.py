"""The domain means psiC of runs merged into one launch: their partial sums are
added in the order the run alone adds them, also where a mode has more partial
sums than a CTA of the inverse DST has threads -- so psi is the run alone's to
the bit, whatever else is in the launch."""
import numpy as np
import pytest

import pequod_b200 as pq
from pequod_b200.workloads import double_gyre

pytestmark = pytest.mark.gpu

# ii, jj, layers, members: partial sums per mode ceil((ii - 2) / 4) above the
# layers * 32 (or * 64) threads; one run's rows below 592 CTAs, the merged above.
SHAPES = [(513, 513, 3, 2), (257, 257, 1, 3), (513, 401, 2, 2), (1025, 301, 3, 3), (513, 601, 3, 2)]


def cfg_ics(ii, jj, L, n, precision):
    cfg = double_gyre(ii, L, 900.0, precision, jj=jj)
    return cfg, [pq.make_ic(ii, jj, L, seed=40 + k, amplitude=1e-7 * cfg.t_scale, sigma=2.0) for k in range(n)]


def alone(cfg, ic, steps):
    m = pq.Model(cfg)
    m.init_perturb(ic)
    m.step(steps)
    psi = m.get("psi")[1:-1, 1:-1, :]
    m.close()
    return psi


@pytest.mark.parametrize("precision", [pq.PREC_FP64, pq.PREC_MIXED])
@pytest.mark.parametrize("ii,jj,L,n", SHAPES)
def test_server_runs_equal_alone(ii, jj, L, n, precision):
    cfg, ics = cfg_ics(ii, jj, L, n, precision)
    srv = pq.Server(16 << 30)
    ids = [srv.submit(cfg, ic, 3) for ic in ics]
    srv.run_until_done(max_steps=3)
    for rid, ic in zip(ids, ics):
        psi, _ = srv.collect(rid)
        assert np.array_equal(psi, alone(cfg, ic, 3))
    srv.close()
