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
        # single-precision rounding (6e-8) amplified by the conditioning of the equilibrated system (about 1e4)
        assert err <= 1e-3, (nrhs, err)
        assert torch.equal(x[sw.mask == 0], torch.zeros_like(x[sw.mask == 0]))
