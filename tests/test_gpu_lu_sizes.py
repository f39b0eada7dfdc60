"""The multifrontal LU over front sizes on both sides of its blocks (32-column steps, 64-entry tiles, 128-column
outer blocks, 256-row inverses) and over the right-hand-side counts of the solve's dispatch."""
import numpy as np
import pytest
import torch

from emerge_b200 import problems
from emerge_b200.direct import DeviceLU
from emerge_b200.sweep import FrequencySweep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def box(cuda):
    P = problems.cavity(n=4, seed=2)
    sw = FrequencySweep(P)
    f = float(P.freqs[50])
    lu0 = DeviceLU(sw)
    K = torch.zeros((sw.n, sw.n), dtype=torch.complex128, device=sw.device)
    rows = torch.repeat_interleave(torch.arange(sw.n, device=sw.device), (sw.plan.indptr[1:] - sw.plan.indptr[:-1]).long())
    K[rows, sw.plan.indices.long()] = lu0.operator_values(f)
    free = torch.nonzero(sw.mask).reshape(-1)
    Kf = K[free][:, free]
    return sw, f, free, Kf


# leaf sizes from a tree of many fronts of a few columns to one front of the whole box (more than 2 000 columns)
@pytest.mark.parametrize("leaf", [1, 6, 40, 100, 1000])
@pytest.mark.parametrize("precision", ["c64", "c128"])
def test_lu_matches_dense_solve(box, leaf, precision):
    sw, f, free, Kf = box
    lu = DeviceLU(sw, leaf_tets=leaf, precision=precision).factor(f)
    g = torch.Generator(device="cpu").manual_seed(leaf)
    for nrhs in (1, 2, 3, 5, 8, 11, 16, 17, 33):
        b = torch.zeros((sw.n, nrhs), dtype=torch.complex128, device=sw.device)
        b[free] = torch.complex(torch.randn(len(free), nrhs, generator=g, dtype=torch.float64),
                                torch.randn(len(free), nrhs, generator=g, dtype=torch.float64)).to(sw.device)
        x = lu.solve(b)
        xd = torch.linalg.solve(Kf, b[free])
        err = (torch.linalg.norm(x[free] - xd, dim=0) / torch.linalg.norm(xd, dim=0)).max().item()
        # single-precision rounding (6e-8) amplified by the equilibrated system: twice the worst that substitution in
        # 32-row steps gives over these leaf sizes (8.7e-5 with complex64 fronts, 2.5e-5 with complex128 ones)
        assert err <= (1.8e-4 if precision == "c64" else 5.2e-5), (nrhs, err)
        assert torch.equal(x[sw.mask == 0], torch.zeros_like(x[sw.mask == 0]))


# error and residual of one solve: twice what substitution in 32-row steps gives (measured: error 3.6e-5 and 1.3e-5 on
# the cavity in complex64 and complex128 fronts, residual 1.5e-4 and 6.5e-5; residual 0.040 and 0.030 on the substrate,
# whose equilibrated system at 1 GHz is near-singular)
@pytest.mark.parametrize("family,precision,err_max,res_max", [("cavity", "c64", 7e-5, 3e-4), ("cavity", "c128", 2.6e-5, 1.3e-4),
                                                              ("substrate", "c64", None, 0.08), ("substrate", "c128", None, 0.06)])
def test_block_inverses_are_as_accurate_as_substitution(cuda, family, precision, err_max, res_max):
    P = problems.cavity(n=5) if family == "cavity" else problems.substrate_box(nx=8, ny=6, nz=6)
    f = float(P.freqs[50]) if family == "cavity" else 1e9
    sw = FrequencySweep(P)
    lu = DeviceLU(sw, precision=precision).factor(f)
    K = torch.zeros((sw.n, sw.n), dtype=torch.complex128, device=sw.device)
    rows = torch.repeat_interleave(torch.arange(sw.n, device=sw.device), (sw.plan.indptr[1:] - sw.plan.indptr[:-1]).long())
    K[rows, sw.plan.indices.long()] = lu.operator_values(f)
    free = torch.nonzero(sw.mask).reshape(-1)
    Kf = K[free][:, free]
    g = torch.Generator(device="cpu").manual_seed(1)
    b = torch.complex(torch.randn(len(free), 4, generator=g, dtype=torch.float64),
                      torch.randn(len(free), 4, generator=g, dtype=torch.float64)).to(sw.device)
    rhs = torch.zeros((sw.n, 4), dtype=torch.complex128, device=sw.device)
    rhs[free] = b
    x = lu.solve(rhs)[free]
    res = (torch.linalg.norm(b - Kf @ x, dim=0) / torch.linalg.norm(b, dim=0)).max().item()
    assert res <= res_max
    if err_max is not None:
        xd = torch.linalg.solve(Kf, b)
        assert (torch.linalg.norm(x - xd, dim=0) / torch.linalg.norm(xd, dim=0)).max().item() <= err_max
