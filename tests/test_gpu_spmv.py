"""The sweep SpMV on CSR matrices without the DOF-pair structure: odd sizes, empty and masked rows, rows
longer than one index chunk, every batch width of the kernel's dispatch, with and without B."""
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
