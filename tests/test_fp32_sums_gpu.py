"""The FP32 iteration's running sums.  A constant vector on a uniform periodic box: every thread of the
sum w r r adds equal terms, whose roundings all go the same way.  A chain of n equal terms
c is off by at most sum_k 2^-24 k c = n / 2 2^-24 of its total; at 60 x 72 x 64 elements of order 7 a
chain has 228 terms (4 components of a vector, 608 blocks of 256 threads, 142 M nodes): 6.8e-6
(four times as long, as one chain over the vector's components, it is 1.15e-5 off).  The other sum of the step, p . A p, is over 8 to 16 nodes and then in FP64: 16 * 2^-24 for it and the
roundings of the operator and the scaling together, 1e-6."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_one_step_of_a_constant(nb, dev):
    bp = nb.BP(7, 60, 72, 64, periodic=True, dirichlet=False, perturb=0.0)
    lam = torch.ones(2 * bp.Nlocal, dtype=torch.float64, device=dev)
    step = []
    for solver in (nb.SOLVER_FP64, nb.SOLVER_MIXED):
        r = torch.ones(bp.Nlocal, dtype=torch.float64, device=dev)
        x = torch.zeros_like(r)
        bp.pcg(lam, r, x, 1e-8, 1, solver=solver, precond=nb.PRECOND_COPY, fixed_iterations=True)
        step.append(float(x.mean()))
    assert step[0] > 0
    assert abs(step[1] - step[0]) <= 7.8e-6 * step[0]
