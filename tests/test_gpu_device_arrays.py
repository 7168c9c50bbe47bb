"""Device arrays solved in place (pq_helm, pq_batch_helm) give the host path's
bits, boundary values included; batches past one copy launch's members."""
import ctypes as C

import numpy as np
import pytest

import pequod_b200 as pq

pytestmark = pytest.mark.gpu


def on_device(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda()


def ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def helm_cfg(ii, jj, ss, periodic, precision):
    d = pq.ModelDesc()
    d.ii, d.jj, d.layers, d.periodic_j, d.precision = ii, jj, len(ss), int(periodic), precision
    d.limiter, d.bc_type, d.dt = 1, pq.BC_FREE_SLIP, 1.0
    for k in range(len(ss)):
        d.ss[k], d.h[k] = ss[k], 1.0
        d.m2z[k + len(ss) * k] = d.z2m[k + len(ss) * k] = 1.0
    return pq.Config(d, None, 1.0)


@pytest.mark.parametrize("precision", [pq.PREC_FP64, pq.PREC_MIXED])
@pytest.mark.parametrize("ii,jj,L,periodic", [(5, 5, 1, False), (9, 7, 3, False), (17, 40, 2, True), (65, 33, 5, False),
                                              (129, 70, 8, False), (513, 9, 2, True), (1025, 6, 1, False)])
def test_helm_in_place(ii, jj, L, periodic, precision):
    import torch

    m = pq.Model(helm_cfg(ii, jj, [0.01 * k for k in range(L)], periodic, precision))
    z = np.asfortranarray(np.random.default_rng(ii + jj).standard_normal((ii, jj, L)))
    want = m.helm(z)
    d = on_device(z)
    torch.cuda.synchronize()
    assert pq.lib().pq_helm(m.ctx, ptr(d), pq.PTR_DEVICE) == pq.PQ_OK
    assert np.array_equal(d.cpu().numpy().transpose(2, 1, 0), want)
    m.close()


@pytest.mark.parametrize("n", [1, 3, 257])
def test_batch_of_device_arrays(n):
    import torch

    rng = np.random.default_rng(n)
    shapes = [(int(rng.choice((5, 9, 17, 33))), int(rng.integers(5, 40)), int(rng.integers(1, 4))) for _ in range(n)]
    b = pq.Batch(shapes, [rng.uniform(0.0, 1.0, s[2]) for s in shapes])
    rhs = [np.asfortranarray(rng.standard_normal(s)) for s in shapes]
    want = b.helm(rhs)
    d = [on_device(r) for r in rhs]
    torch.cuda.synchronize()
    ptrs = (C.POINTER(C.c_double) * n)(*[ptr(t) for t in d])
    assert pq.lib().pq_batch_helm(b.ctx, ptrs, pq.PTR_DEVICE) == pq.PQ_OK
    assert all(np.array_equal(t.cpu().numpy().transpose(2, 1, 0), w) for t, w in zip(d, want))
    b.close()
