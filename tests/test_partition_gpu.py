"""An element's result does not depend on the other elements of the call, bit for bit: not on
their number, which chooses the kernel's launch shape, and not on their values."""
import numpy as np
import pytest
import torch

from test_axhelm_gpu import T

pytestmark = pytest.mark.gpu


def problem(O, N, E, nf=1, seed=11):
    m = O.BoxMesh(N, E, 1, 1, perturb=0.1, seed=seed)
    L = m.Nlocal
    lam = np.concatenate([O.uniform(L, seed, 1, 0.5, 1.5), O.uniform(L, seed, 2, 0.5, 2.0)])
    return m, lam, O.uniform(nf * L, seed, 3, -1, 1)


@pytest.mark.parametrize("N,E", [(1, 40), (2, 15), (3, 9), (4, 11), (5, 1500), (6, 1100)])
@pytest.mark.parametrize("bad", [np.inf, 1e-310])
def test_fp64_neighbours_of_an_element_without_a_fixed_point_form(nb, O, dev, N, E, bad):
    """Several elements share a CTA at these orders; one of them takes the FP64 sums."""
    m, lam, q = problem(O, N, E)
    Np = (N + 1) ** 3

    def run():
        Aq = torch.full((m.Nlocal,), 7.0, dtype=torch.float64, device=dev)
        nb.axhelm(N + 1, 0, nb.FP64, E, m.Nlocal, T(m.ggeo, dev), T(m.D, dev), T(lam, dev), T(q, dev), Aq)
        return Aq.cpu().numpy().reshape(E, Np)

    a = run()
    for e in (0, E // 2, E - 1):
        keep = q[e * Np:(e + 1) * Np].copy()
        if np.isinf(bad):
            q[e * Np + 2] = bad
        else:
            q[e * Np:(e + 1) * Np] = 0
            q[e * Np + 2] = bad
        assert np.array_equal(np.delete(run(), e, 0), np.delete(a, e, 0))
        q[e * Np:(e + 1) * Np] = keep
