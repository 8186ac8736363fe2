"""A solve whose operator is not positive ends in its first step: the status says so, r and x are left
as they were, and the next solve on the same handle is a good one.  (The launch that finds it out
also assembles A p; the end of the solve is for the launches after it.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,box,nf", [(3, (3, 2, 2), 1), (7, (4, 4, 4), 1), (7, (11, 11, 11), 1), (7, (4, 4, 4), 3)])
@pytest.mark.parametrize("use_graph", [True, False])
def test_breakdown_in_the_first_step(nb, dev, N, box, nf, use_graph):
    bp = nb.BP(N, *box, Nfields=nf, perturb=0.1, seed=2)
    n = nf * bp.Nlocal
    g = torch.Generator(device=dev).manual_seed(N)
    f = torch.rand(n, dtype=torch.float64, device=dev, generator=g) - 0.5
    bp.ogs.gather_scatter_many(f, nf, bp.Nlocal)
    good = torch.ones(2 * bp.Nlocal, dtype=torch.float64, device=dev)
    sols = []
    for lam in (good, -good, good, -good, good):
        r, x = f.clone(), torch.zeros_like(f)
        st = bp.pcg(lam, r, x, 1e-9, 2000, solver=nb.SOLVER_MIXED, precond=nb.PRECOND_COPY, use_graph=use_graph)
        if lam is good:
            assert st["status"] == 0 and st["true_rel_res"] <= 1e-9
            sols.append(x.clone())
        else:
            assert st["status"] == nb.ERR_BREAKDOWN and not x.any()
    assert torch.equal(sols[0], sols[1]) and torch.equal(sols[0], sols[2])
