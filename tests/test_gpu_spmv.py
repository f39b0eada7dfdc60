"""The sweep SpMV on CSR matrices without the DOF-pair structure: odd sizes, empty and masked rows, rows
longer than one index chunk, every batch width of the kernel's dispatch, with and without B."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from emerge_b200 import _lib
from emerge_b200._lib import Handle, lib, ptr

pytestmark = pytest.mark.gpu


def _csr(n, seed, paired):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, min(n, 110), n)
    lens[:3] = [0, 1, 33][:n] if n > 33 else [1, 0, 1][:n]
    rows = [np.sort(rng.choice(n, k, replace=False)) for k in lens]
    if paired:                                  # rows i and i + n/2 share their columns, as a mesh entity's do
        for i in range(n // 2):
            rows[i + n // 2] = rows[i]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    idx = (np.concatenate(rows) if indptr[-1] else np.zeros(0)).astype(np.int32)
    c = lambda: rng.standard_normal(len(idx)) + 1j * rng.standard_normal(len(idx))
    return indptr, idx, c(), c(), rng


@pytest.mark.parametrize("n,paired", [(1, False), (2, True), (37, False), (300, True), (301, False)])
@pytest.mark.parametrize("S", [1, 2, 4, 8, 16, 32, 64, 128])
@pytest.mark.parametrize("has_b", [True, False])
def test_spmv_matches_scipy(cuda, n, paired, S, has_b):
    indptr, idx, ev, bv, rng = _csr(n, 7 * n + S, paired)
    mask = (rng.random(n) > 0.1).astype(np.uint8)
    x = rng.standard_normal((n, S)) + 1j * rng.standard_normal((n, S))
    k2 = rng.uniform(0.5, 2.0, S)
    np_rows = np.arange(0, n, 3)
    pcols = rng.integers(0, n, 5 * len(np_rows)).astype(np.int32)
    pvals = rng.standard_normal(len(pcols)) + 1j * rng.standard_normal(len(pcols))
    pport = rng.integers(0, 2, len(pcols)).astype(np.int32)
    gam = rng.standard_normal((S, 2)) + 1j * rng.standard_normal((S, 2))
    E, B = (sp.csr_matrix((v, idx, indptr), shape=(n, n)) for v in (ev, bv))
    ref = E @ x - (B @ x) * k2 * has_b
    mag = abs(E) @ np.abs(x) + (abs(B) @ np.abs(x)) * k2
    for i, r in enumerate(np_rows):
        for j in range(5 * i, 5 * i + 5):
            t = gam[:, pport[j]] * pvals[j] * x[pcols[j]]
            ref[r] += t
            mag[r] += np.abs(t)
    ref[mask == 0] = 0
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(cuda, t)
    c128, i32 = torch.complex128, torch.int32
    # (the library rejects null matrices: an empty one gets a dummy entry)
    dev = [d(indptr, i32), d(idx if len(idx) else [0], i32), d(ev if len(ev) else [0], c128),
           d(bv if len(bv) else [0], c128) if has_b else None]
    k2d, gd = d(k2, torch.float64), d(gam, c128)
    pr, pp = d(np_rows, i32), d(5 * np.arange(len(np_rows) + 1), i32)
    pc, pv, po, md, xd = d(pcols, i32), d(pvals, c128), d(pport, i32), d(mask, torch.uint8), d(x, c128)
    h = Handle.get(cuda)
    for fn in (lib().emfem_sweep_spmv, lib().emfem_sweep_spmv_noalloc):
        y = torch.full((n, S), complex(np.nan, np.nan), dtype=c128, device=cuda)
        st = fn(h.h, n, ptr(dev[0]), ptr(dev[1]), ptr(dev[2]), ptr(dev[3]), S, ptr(k2d), len(np_rows), ptr(pr),
                ptr(pp), ptr(pc), ptr(pv), ptr(po), 2, ptr(gd), ptr(md), ptr(xd), ptr(y))
        assert st == 0, _lib.last_error()
        err = np.abs(y.cpu().numpy() - ref)
        # at most 115 terms a row, a few roundings per term: 256 eps of the summed magnitudes
        assert (err <= 256 * np.finfo(float).eps * mag + 1e-300).all(), (err / (mag + 1e-300)).max()


@pytest.mark.parametrize("S", [1, 8, 32])
def test_patch_entries_of_other_ports_are_left_out(cuda, S):
    """A call over the first n_ports ports of a patch that lists more: entries of the others do not count, in the
    products and in the preconditioner blocks of a solve."""
    n, nports = 64, 2
    rng = np.random.default_rng(S)
    A = sp.random(n, n, 0.2, random_state=5, format="csr") + sp.diags(np.full(n, 8.0))
    A = (A + 1j * sp.diags(rng.random(n))).tocsr()
    A.sort_indices()
    prow = np.arange(0, n, 2)
    pcols = np.stack([prow, prow, prow, prow], 1).reshape(-1)               # on the diagonal, four ports a row
    pport = np.tile([0, 1, 5, -1], len(prow))
    pvals = rng.standard_normal(len(pcols)) + 1j * rng.standard_normal(len(pcols))
    gam = 0.5 * (rng.standard_normal((S, nports)) + 1j * rng.standard_normal((S, nports)))
    x = rng.standard_normal((n, S)) + 1j * rng.standard_normal((n, S))
    ref = A @ x
    for i, j, q, v in zip(np.repeat(prow, 4), pcols, pport, pvals):
        if 0 <= q < nports:
            ref[i] += gam[:, q] * v * x[j]
    d = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to(cuda, t)
    c128, i32 = torch.complex128, torch.int32
    ip, ix, ev = d(A.indptr, i32), d(A.indices, i32), d(A.data, c128)
    pr, pp, pc, pv, po = d(prow, i32), d(4 * np.arange(len(prow) + 1), i32), d(pcols, i32), d(pvals, c128), d(pport, i32)
    k2, gd, md, xd = (d(np.ones(S), torch.float64), d(gam, c128), d(np.ones(n), torch.uint8), d(x, c128))
    h = Handle.get(cuda)
    for fn in (lib().emfem_sweep_spmv, lib().emfem_sweep_spmv_noalloc):
        y = torch.empty_like(xd)
        st = fn(h.h, n, ptr(ip), ptr(ix), ptr(ev), None, S, ptr(k2), len(prow), ptr(pr), ptr(pp), ptr(pc), ptr(pv),
                ptr(po), nports, ptr(gd), ptr(md), ptr(xd), ptr(y))
        assert st == 0, _lib.last_error()
        np.testing.assert_allclose(y.cpu().numpy(), ref, rtol=0, atol=1e-12 * np.abs(ref).max())
    sz = ctypes.c_size_t()
    nnz = len(A.data)
    assert lib().emfem_krylov_workspace_size(n, nnz, S, 0, ctypes.byref(sz)) == 0
    ws = torch.empty(sz.value, dtype=torch.uint8, device=cuda)
    ga = np.ascontiguousarray(np.stack([gam.real, gam.imag], -1).reshape(-1))
    status, iters, rel = (ctypes.c_int * S)(), (ctypes.c_int * S)(), (ctypes.c_double * S)()
    xs, b = torch.zeros_like(xd), d(ref, c128)
    st = lib().emfem_krylov_solve(h.h, 1, n, nnz, ptr(ip), ptr(ix), ptr(ev), None, S, (ctypes.c_double * S)(*np.ones(S)),
                                  len(prow), ptr(pr), ptr(pp), ptr(pc), ptr(pv), ptr(po), nports,
                                  (ctypes.c_double * len(ga))(*ga), ptr(md), ptr(b), ptr(xs), 1e-12, 500, 1, 0, ptr(ws),
                                  ws.numel(), status, iters, rel, None)
    assert st == 0, _lib.last_error()
    np.testing.assert_allclose(xs.cpu().numpy(), x, rtol=0, atol=1e-9 * np.abs(x).max())
