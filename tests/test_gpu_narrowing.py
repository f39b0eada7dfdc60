"""A batch whose systems converge at different iterations is narrowed while it runs; every system must come back
in its own column, with its own status and iteration count."""
import numpy as np
import pytest
import torch

from emerge_b200 import problems
from emerge_b200.sweep import FrequencySweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsys,precond,maxit", [(13, "aux", 20000), (32, "aux", 20000), (16, "none", 40), (24, "aux", 150),
                                                (7, "aux", 150)])
def test_narrowed_batch_solves_every_column(cuda, nsys, precond, maxit):
    P = problems.waveguide(nx=10, ny=5, nz=20)            # n * nsys beyond the width from which batches are narrowed
    sw = FrequencySweep(P)
    assert sw.n * nsys >= 1 << 18
    freqs = np.linspace(7.2e9, 12.5e9, nsys)
    systems = [(float(f), k % 2) for k, f in enumerate(freqs)]
    b = sw.rhs(systems)
    b[:, 2] = 0                                            # one system that is solved before it starts
    k0, gam = sw.k0sq(freqs), sw.gammas(freqs)
    tol = 1e-9
    res = sw.solve_rhs(k0, b, gam, tol=tol, maxit=maxit, precond=precond)
    assert res.iters[2] == 0 and res.status[2] == 0 and torch.count_nonzero(res.x[:, 2]) == 0
    y = sw.apply(systems, res.x)
    bm = b * sw.mask[:, None]
    nb = torch.linalg.norm(bm, dim=0)
    rel = (torch.linalg.norm(bm - y, dim=0) / torch.where(nb > 0, nb, torch.ones_like(nb))).cpu().numpy()
    np.testing.assert_allclose(rel, res.relres, rtol=1e-3, atol=1e-13)
    if maxit >= 20000:
        assert (res.status == 0).all() and (rel <= tol).all()
        assert len(set(res.iters.tolist())) > 3            # the systems stop at different iterations
    else:
        live = np.arange(nsys) != 2
        assert (res.status[live] == 1).any() and (res.iters <= maxit).all()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_repeated_solves_give_the_same_bits(cuda, precision):
    """When the batch narrows is decided from the iteration counts, not from how far the host has come."""
    sw = FrequencySweep(problems.waveguide(nx=10, ny=5, nz=20))
    systems = [(float(f), k % 2) for k, f in enumerate(np.linspace(7.2e9, 12.5e9, 16))]
    assert sw.n * len(systems) >= 1 << 18
    runs = [sw.solve(systems, tol=1e-8, maxit=20000, precond="aux", precision=precision) for _ in range(4)]
    assert (runs[0].status == 0).all()
    for r in runs[1:]:
        assert torch.equal(r.x, runs[0].x) and np.array_equal(r.iters, runs[0].iters)


@pytest.mark.parametrize("precond,maxit,nsys", [("block_jacobi", 200, 16), ("block_jacobi", 200, 32), ("aux", 150, 16),
                                                ("aux", 150, 32), ("learned", 60, 16), ("learned", 60, 32),
                                                ("lu", 12, 7), ("lu", 12, 16), ("lu", 12, 32)])
def test_bits_do_not_depend_on_the_other_columns(cuda, precond, maxit, nsys):
    """Three systems among live neighbours (the batch keeps its width) and among columns that stop at once (it is
    narrowed after the first replay, or the LU applied to some of its columns): the same sums in the same order."""
    from emerge_b200.auxspace import Network
    sw = FrequencySweep(problems.waveguide(nx=10, ny=5, nz=20))
    assert sw.n * nsys >= 1 << 18
    freqs = np.linspace(8.2e9, 11.5e9, nsys)
    systems = [(float(f), k % 2) for k, f in enumerate(freqs)]
    kw = dict(tol=1e-13, maxit=maxit)
    if precond == "learned":
        net = Network(sw.aux_space(), seed=4, init="random")
        net.params.mul_(0.5)
        sw.set_network(net)
    if precond == "lu":
        kw["lu"] = sw.direct_solver().factor(float(freqs[nsys // 2]))
    else:
        kw["precond"] = precond
    b = sw.rhs(systems)
    live = [1, 6, nsys - 5]                  # (none at the LU's own frequency)
    alone = torch.zeros_like(b)
    alone[:, live] = b[:, live]
    full, few = (sw.solve_rhs(sw.k0sq(freqs), v, sw.gammas(freqs), **kw) for v in (b, alone))
    assert torch.equal(full.x[:, live], few.x[:, live])
    assert np.array_equal(full.iters[live], few.iters[live]) and (few.iters[live] > 2).all()
