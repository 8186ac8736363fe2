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


def line_nodes(Nq, nf, bk, trilinear):
    """Nodes from which the FP32 forms run by lines (the larger of FP32's and BF16's)."""
    if not bk and nf == 1:
        return 1200000 if trilinear else 4200000 if Nq == 6 or (Nq >= 8 and Nq != 11) else 2000000 if Nq == 4 else 1000000
    return 2000000 if not bk and Nq == 4 and not trilinear else 600000


def whole_and_chunks(nb, N, E, flags, prec, per_element, g, D, lam, q, cuts):
    """The operator in one call and element range by element range."""
    Np, L = (N + 1) ** 3, E * (N + 1) ** 3
    whole, parts = torch.full_like(q, 7.0), torch.full_like(q, 8.0)
    nb.axhelm(N + 1, flags, prec, E, L, g, D, lam, q, whole)
    ends = [0] + [c for c in cuts if c < E] + [E]
    for a, b in zip(ends, ends[1:]):
        nb.axhelm(N + 1, flags, prec, b - a, L, g[a * per_element:], D, None if lam is None else lam[a * Np:], q[a * Np:],
                  parts[a * Np:])
    assert torch.equal(whole, parts)


@pytest.mark.parametrize("N", [3, 5, 7, 8, 11])
@pytest.mark.parametrize("flags", [0, 1, 2, 3])
@pytest.mark.parametrize("form", ["FP32", "BF16", "FP32_TRILINEAR"])
def test_fp32_forms_by_lines_and_by_columns(nb, O, dev, N, flags, form):
    Nq, Np, prec = N + 1, (N + 1) ** 3, getattr(nb, form)
    nf = 3 if flags & nb.AX_N3 else 1
    E = -(-line_nodes(Nq, nf, flags & nb.AX_BK, prec == nb.FP32_TRILINEAR) // Np) + 1
    m, lam, q = problem(O, N, E, nf)
    F = torch.float32
    if prec == nb.FP32_TRILINEAR:
        g, per = torch.zeros(24 * E, dtype=F, device=dev), 24
        nb.trilinear_coeffs(E, T(m.EX, dev), T(m.EY, dev), T(m.EZ, dev), g)
    else:
        g, per = T(m.ggeo, dev, torch.bfloat16 if prec == nb.BF16 else F), 7 * Np
    lam = None if flags & nb.AX_BK else T(lam, dev, torch.bfloat16 if prec == nb.BF16 else F)
    whole_and_chunks(nb, N, E, flags, prec, per, g, T(m.D, dev, F), lam, T(q, dev, F), [1, E // 3, E // 2])


@pytest.mark.parametrize("N,E", [(1, 700), (3, 800), (4, 2400), (5, 1400), (6, 6000), (7, 1600), (8, 650), (13, 300)])
@pytest.mark.parametrize("flags", [0, 3])
@pytest.mark.parametrize("form", ["FP64", "FP64_SPLIT"])
def test_fp64_forms(nb, O, dev, N, E, flags, form):
    """Across the line between three groups of threads per element and one (FP64)."""
    if form == "FP64_SPLIT" and N > 11:
        pytest.skip("built for N <= 11")
    m, lam, q = problem(O, N, E, 3 if flags & nb.AX_N3 else 1)
    lam = None if flags & nb.AX_BK else T(lam, dev)
    whole_and_chunks(nb, N, E, flags, getattr(nb, form), 7 * (N + 1) ** 3, T(m.ggeo, dev), T(m.D, dev), lam, T(q, dev),
                     [2, E // 8, E // 2])
