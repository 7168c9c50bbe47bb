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


@pytest.mark.parametrize("where", ["misaligned", "null", "shared"])
def test_arrays_the_kernels_do_not_address(where):
    """Arrays that take the copies instead: the same results, the same refusals."""
    import torch

    shapes = [(17, 9, 1), (17, 9, 1)]
    b = pq.Batch(shapes, [np.array([0.1]), np.array([0.1])])
    rng = np.random.default_rng(5)
    rhs = [np.asfortranarray(rng.standard_normal(s)) for s in shapes]
    want = b.helm(rhs)
    n = 17 * 9
    host = np.concatenate([r.transpose(2, 1, 0).ravel() for r in rhs])
    raw = torch.zeros(16 * n + 8, dtype=torch.uint8, device="cuda")
    off = 4 if where == "misaligned" else 0
    raw[off : off + 16 * n] = torch.from_numpy(host.view(np.uint8)).cuda()
    torch.cuda.synchronize()
    second = 0 if where == "shared" else 8 * n
    at = [raw.data_ptr() + off, raw.data_ptr() + off + second]
    if where == "null":  # refused
        at[1] = None
    ptrs = (C.POINTER(C.c_double) * 2)(*[C.cast(C.c_void_p(a), C.POINTER(C.c_double)) for a in at])
    rc = pq.lib().pq_batch_helm(b.ctx, ptrs, pq.PTR_DEVICE)
    if at[1] is None:
        assert rc != pq.PQ_OK
    else:
        assert rc == pq.PQ_OK
        got = np.frombuffer(raw.cpu().numpy()[off : off + 16 * n].tobytes(), dtype=np.float64)
        assert np.array_equal(got[:n].reshape(1, 9, 17).transpose(2, 1, 0), want[0])
        if where == "misaligned":
            assert np.array_equal(got[n:].reshape(1, 9, 17).transpose(2, 1, 0), want[1])
    b.close()
