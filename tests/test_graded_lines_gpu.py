"""The fixed-point contractions (csrc/fixedpt.cuh) on values that are graded along a line, against
extended precision (np.longdouble) on the same operands, component by component.

A contraction's result is off by at most (Nq + 2) 2^-54 of max|D| max|v| of its row and line.
Where the full-length form is taken (Nq <= 5, or a D without centro-antisymmetry) that is
Nq (2^-56 + 2^-58) + 2^-57, 9.4e-17 at Nq = 5, and a line with a row whose terms are below 2^-9
max|D| max|v| goes to the FP64 sums.  So each of the operator's two contractions is off by at
most 9.4e-17 * 2^9 = 4.8e-14 of its terms, the rest by a few 2^-53: below 1.3e-13."""
import numpy as np
import pytest
import torch

from test_axhelm_gpu import T

pytestmark = pytest.mark.gpu

LD = np.longdouble


def contract(D, v):
    """D along r, s, t of v[..., k, j, i]."""
    return (np.einsum("im,ekjm->ekji", D, v), np.einsum("jm,ekmi->ekji", D, v), np.einsum("km,emji->ekji", D, v))


def back(D, r, s, t):
    return np.einsum("mi,ekjm->ekji", D, r) + np.einsum("mj,ekmi->ekji", D, s) + np.einsum("mk,emji->ekji", D, t)


def mix(g, q):
    G = [g[:, k] for k in range(7)]
    return (G[1] * q[0] + G[2] * q[1] + G[3] * q[2], G[2] * q[0] + G[4] * q[1] + G[5] * q[2],
            G[3] * q[0] + G[5] * q[1] + G[6] * q[2])


def operator(D, g, l0, l1, q):
    """The result and the sum of the magnitudes of its terms."""
    out = back(D, *(l0 * v for v in mix(g, contract(D, q)))) + g[:, 0] * l1 * q
    D, g, q = abs(D), abs(g), abs(q)
    return out, back(D, *(l0 * v for v in mix(g, contract(D, q)))) + g[:, 0] * l1 * q


def run(nb, dev, N, E, D, g, lam, q):
    Aq = torch.full((q.size,), 7.0, dtype=torch.float64, device=dev)
    nb.axhelm(N + 1, 0, nb.FP64, E, q.size, *(T(a.ravel(), dev) for a in (g, D, lam, q)), Aq)
    return Aq.cpu().numpy().reshape(q.shape)


def problem(O, N, E, kind, seed):
    rng = np.random.default_rng([N, E, seed])
    n = N + 1
    m = O.BoxMesh(N, E, 1, 1, perturb=0.1, seed=3)
    D, g = np.asarray(m.D).reshape(n, n), np.asarray(m.ggeo).reshape(E, 7, n, n, n)
    shape = (E, n, n, n)
    lam, q = rng.uniform(0.5, 1.5, (2,) + shape), rng.uniform(-1, 1, shape)
    for e in range(E):
        at = tuple(rng.integers(0, n, 3))
        if kind == "lambda spike":
            lam[0, e][at] *= 1e12
        elif kind == "lambda graded":
            lam[0, e] *= 2.0 ** rng.uniform(-40, 0, (n, n, n))
        elif kind == "q spike":
            q[e][at] *= 1e12
        elif kind == "steep":
            x = (np.asarray(O.gll(N)[0]) + 1) / 2
            q[e] = np.exp(-20 * x) * rng.uniform(0.9, 1.1, (n, n, n))
    return D, g, lam, q


@pytest.mark.parametrize("N", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["lambda spike", "lambda graded", "q spike", "steep"])
def test_low_orders_component_by_component(nb, O, dev, N, kind):
    E = 25
    D, g, lam, q = problem(O, N, E, kind, 1)
    ref, terms = operator(*(a.astype(LD) for a in (D, g, lam[0], lam[1], q)))
    got = run(nb, dev, N, E, D, g, lam, q)
    assert np.all(abs(got - ref) <= 1.3e-13 * terms)


@pytest.mark.parametrize("N", [4, 6, 7, 9])
@pytest.mark.parametrize("kind", ["lambda spike", "q spike", "banded"])
def test_any_matrix_component_by_component(nb, O, dev, N, kind):
    """Without the symmetry of nodes about the centre: one-sided node sets keep every entry
    beside the diagonal in range; a banded matrix, of mostly zeros, takes the FP64 sums, whose
    2 Nq + 20 roundings are within 1e-14 of the terms."""
    E, n = 7, N + 1
    D, g, lam, q = problem(O, N, E, "lambda graded" if kind == "banded" else kind, 2)
    if kind == "banded":
        D = np.diag(np.ones(N), 1) - np.diag(np.ones(N), -1) + 0.25 * np.diag(np.arange(n) % 2)
        q *= 2.0 ** np.random.default_rng(N).uniform(-40, 0, q.shape)
    else:
        D = D * np.linspace(1.0, 1.5, n)[:, None]
    ref, terms = operator(*(a.astype(LD) for a in (D, g, lam[0], lam[1], q)))
    got = run(nb, dev, N, E, D, g, lam, q)
    # lines that are not looked at: rows of D up to 2^6 apart in their entries, values 2^4:
    # 12 * 2^-54 * 2^(6 + 4) = 6.8e-13, twice
    assert np.all(abs(got - ref) <= (1e-14 if kind == "banded" else 1.4e-12) * terms)


@pytest.mark.parametrize("N", [5, 6, 7, 8, 10, 11, 13])
@pytest.mark.parametrize("E", [3, 1501])
def test_even_odd_within_its_line_bound(nb, O, dev, N, E):
    """Steep lines in the even-odd form: (Nq + 2) 2^-54 max|D| max|v| of each line, the first
    contraction's share taken through the geometric factors and D^T, and 30 roundings."""
    n = N + 1
    D, g, lam, q = problem(O, N, E, "steep", 3)
    D = (D - D[::-1, ::-1]) / 2  # symmetric to the last bit
    ref, terms = operator(*(a.astype(LD) for a in (D, g, lam[0], lam[1], q)))
    got = run(nb, dev, N, E, D, g, lam, q)
    u, A, l0 = (n + 2) * 2.0 ** -54, abs(D), abs(lam[0])
    row = A.max(1)
    first = (u * row[None, None, None, :] * abs(q).max(3, keepdims=True),
             u * row[None, None, :, None] * abs(q).max(2, keepdims=True),
             u * row[None, :, None, None] * abs(q).max(1, keepdims=True))
    bound = back(A, *(l0 * v for v in mix(abs(g), first)))
    w = [l0 * v for v in mix(abs(g), contract(A, abs(q)))]  # at least the second lines' values
    col = A.max(0)
    bound += u * (col[None, None, None, :] * w[0].max(3, keepdims=True) +
                  col[None, None, :, None] * w[1].max(2, keepdims=True) +
                  col[None, :, None, None] * w[2].max(1, keepdims=True))
    assert np.all(abs(got - ref) <= bound + 30 * 2.0 ** -53 * terms)
