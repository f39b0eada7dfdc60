"""The LU's diagonal blocks with pivots below the floor: every warp of a block must raise them alike, so repeated
factorizations of one matrix agree to the last bit and count the same raised pivots."""
import ctypes

import numpy as np
import pytest
import torch

from emerge_b200._lib import Handle, check, lib, ptr

pytestmark = pytest.mark.gpu


def _fronts(nf, e, b, K):
    """LU handle of nf unconnected fronts of e own and b boundary DOFs, front v holding the dense K[v]."""
    i32 = lambda a: np.ascontiguousarray(a, np.int32)
    n = e + b
    ptrs = np.arange(nf + 1, dtype=np.int64)
    slot = i32(np.arange(nf * n * n).reshape(nf, n, n).transpose(0, 2, 1))        # off = row + column * n
    arrs = [i32(np.full(nf, e)), i32(np.full(nf, b)), i32(np.full(nf, -1)), i32(np.zeros(nf)), ptrs * n,
            i32(np.arange(nf * n)), i32(np.zeros(max(1, nf * b))), ptrs * n * n, slot, i32(np.tile(np.arange(n * n), nf))]
    m = ctypes.c_void_p()
    check(lib().emfem_mf_create(Handle.get(K.device).h, nf * n, nf, *[a.ctypes.data_as(ctypes.c_void_p) for a in arrs],
                                ctypes.byref(m)), "emfem_mf_create")
    return m


@pytest.mark.parametrize("bits", [64, 128])
@pytest.mark.parametrize("tail", [0, 6])
def test_raised_pivots_are_the_same_every_time(cuda, bits, tail):
    rng = np.random.default_rng(bits + tail)
    nf, nblk, e = 300, 2, 64 + tail
    K = np.zeros((nf, e, e), complex)
    live = np.zeros((nf, e), bool)
    for v in range(nf):
        for k in range(nblk):
            q = 32 * k + rng.permutation(32)
            # 16 well-conditioned DOFs, 8 coupled in pairs by entries far below the floor, 8 without any entry
            K[v][np.ix_(q[:16], q[:16])] = (np.eye(16) + 0.1 * rng.standard_normal((16, 16)) / 4
                                            + 0.1j * rng.standard_normal((16, 16)) / 4)
            for a, b in zip(q[16:24:2], q[17:24:2]):
                K[v, a, b] = K[v, b, a] = 1e-9 * (1 + rng.random())
            live[v, q[:16]] = True
        if tail:
            t = slice(64, e)
            K[v, t, t] = np.eye(tail)
            live[v, t] = True
    Kd = torch.from_numpy(K).to(cuda)
    b = rng.standard_normal((nf, e)) + 1j * rng.standard_normal((nf, e))
    bd = torch.from_numpy(b.reshape(-1, 1)).to(cuda)
    m = _fronts(nf, e, 0, Kd)
    try:
        check(lib().emfem_mf_set_precision(m, bits), "emfem_mf_set_precision")
        check(lib().emfem_mf_reserve(m, 1), "emfem_mf_reserve")
        xs = []
        for _ in range(10):
            raised = ctypes.c_int()
            check(lib().emfem_mf_factor(m, ptr(Kd), ctypes.byref(raised)), "emfem_mf_factor")
            assert raised.value == nf * nblk * 16
            xs.append(torch.empty_like(bd))
            check(lib().emfem_mf_solve(m, 1, ptr(bd), ptr(xs[-1])), "emfem_mf_solve")
        assert all(torch.equal(x, xs[0]) for x in xs[1:])
        x = xs[0].cpu().numpy().reshape(nf, e)
        assert np.isfinite(x).all()
        for v in range(0, nf, 37):                 # the well-conditioned DOFs are not coupled to the raised ones
            ref = np.linalg.solve(K[v][np.ix_(live[v], live[v])], b[v, live[v]])
            # factors are complex64 in both precisions; the blocks' condition is below 3
            assert np.linalg.norm(x[v, live[v]] - ref) <= 32 * 6e-8 * 3 * np.linalg.norm(ref)
    finally:
        torch.cuda.synchronize()
        lib().emfem_mf_destroy(m)


def test_boundary_dofs_that_no_front_eliminates_are_zero(cuda):
    """Fronts with a boundary and no parent: the solve takes the boundary as zero, also after solves of other widths."""
    rng = np.random.default_rng(1)
    nf, e, nb = 3, 70, 5
    n = e + nb
    K = np.eye(n) + 0.2 * (rng.standard_normal((nf, n, n)) + 1j * rng.standard_normal((nf, n, n))) / n ** 0.5
    Kd = torch.from_numpy(K).to(cuda)
    m = _fronts(nf, e, nb, Kd)
    try:
        check(lib().emfem_mf_factor(m, ptr(Kd), None), "emfem_mf_factor")
        for nrhs in (16, 3, 1):
            b = rng.standard_normal((nf, n, nrhs)) + 1j * rng.standard_normal((nf, n, nrhs))
            bd = torch.from_numpy(b.reshape(nf * n, nrhs)).to(cuda)
            xd = torch.empty_like(bd)
            check(lib().emfem_mf_solve(m, nrhs, ptr(bd), ptr(xd)), "emfem_mf_solve")
            x = xd.cpu().numpy().reshape(nf, n, nrhs)
            assert (x[:, e:] == 0).all()
            ref = np.linalg.solve(K[:, :e, :e], b[:, :e])
            # complex64 factors of a matrix with condition below 10
            assert np.linalg.norm(x[:, :e] - ref) <= n * 6e-8 * 10 * np.linalg.norm(ref)
    finally:
        torch.cuda.synchronize()
        lib().emfem_mf_destroy(m)
