"""The advection operator's fixed-point contractions (csrc/adv_fx.cuh) where a zero of a matrix
meets values that are far apart along a line, against extended precision (np.longdouble) on the same
operands, component by component.

A contraction is off by at most (cq + 2) 2^-54 of max|M| max|v| of its row and line.  Lines in
which one value is more than 2^(far + 1) above all others (in full rows of the interpolation, where
they are projected) go to the FP64 sums where a row has terms below 2^-9 max|M| max|v|, and entries
of these matrices beside their zeros are within 2^r of their row's largest: cq = 3 (far 10, r 3)
5 2^-54 2^14 = 4.5e-12 of the terms, cq = 12 (6, 10.2) 14 2^-54 2^17.2 = 1.2e-10, the others less; nine
contractions stay below 1.2e-9.  On the element's own nodes there is one contraction, the derivative
(r at most 7): cq = 12 14 2^-54 2^(7 + 7) = 1.3e-11, the others less."""
import numpy as np
import pytest
import torch

from adv_cases import IJW, JW, NVGEO, RX, RY, RZ, SX, SY, SZ, TX, TY, TZ, lagrange

pytestmark = pytest.mark.gpu

LD = np.longdouble


def operator(I, D, u, g, ijw, size=lambda x: x):
    """The operator on longdouble arrays; with size = abs the sum of its terms' magnitudes."""
    I, D, u, g = size(I), size(D), size(u), size(g)
    uc = np.einsum("ai,fecba->fecbi", I, u)
    uc = np.einsum("bj,fecbi->fecji", I, uc)
    uc = np.einsum("ck,fecji->fekji", I, uc)
    d = [np.einsum("in,fekjn->fekji", D, uc), np.einsum("jn,fekni->fekji", D, uc), np.einsum("kn,fenji->fekji", D, uc)]
    hat = [g[:, JW] * (uc[0] * g[:, a] + uc[1] * g[:, b] + uc[2] * g[:, c])
           for a, b, c in ((RX, RY, RZ), (SX, SY, SZ), (TX, TY, TZ))]
    a = sum(h * x for h, x in zip(hat, d))
    a = np.einsum("ck,fekji->fecji", I, a)
    a = np.einsum("bj,fecji->fecbi", I, a)
    return np.einsum("ai,fecbi->fecba", I, a) * ijw


def check(nb, O, dev, nodes, Nq, cq, E, kind, bound):
    rng = np.random.default_rng([Nq, cq, len(kind)])
    xg = O.gll(Nq - 1)[0]
    xc = O.gauss(cq - 1)[0] if nodes == "gauss" else O.gll(cq - 1)[0]
    I, D = lagrange(xg, xc), O.dmatrix(xc).reshape(cq, cq)
    if cq % 2 and Nq % 2:  # the centre to the last bit
        I[:, cq // 2] = 0
        I[Nq // 2, cq // 2] = 1
    U = rng.uniform(-1, 1, (3, E, Nq, Nq, Nq))
    g = rng.uniform(0.5, 1.5, (E, NVGEO, cq, cq, cq))
    vg = rng.uniform(0.5, 1.5, (E, NVGEO, Nq, Nq, Nq))
    mid = cq // 2
    if kind == "metric spike":
        g[:, :, mid, mid, mid] *= 1e6
    elif kind == "metric plane":
        g[:, :, :, :, mid] *= 1e6
    elif kind == "metric ends":
        g[:, :, :, :, [0, -1]] *= 1e6
    elif kind == "velocity spike":
        U[:, :, Nq // 2, Nq // 2, Nq // 2] *= 1e12
    elif kind == "boundary layer":
        U *= (2.0 ** np.linspace(-40, 0, Nq))
    arr = dict(vgeo=vg, cubvgeo=g, cubD=D, cubInterpT=I, U=U)
    t = {k: torch.from_numpy(np.ascontiguousarray(v).ravel()).to(dev) for k, v in arr.items()}
    NU = torch.full((U.size,), 5.0, dtype=torch.float64, device=dev)
    nb.adv_cubature(Nq, cq, E, t["vgeo"], t["cubvgeo"], t["cubD"], t["cubInterpT"], E * Nq ** 3, t["U"], NU)
    got = NU.cpu().numpy().reshape(U.shape)
    a = [x.astype(LD) for x in (I, D, U, g, vg[:, IJW])]
    ref, terms = operator(*a), operator(*a, size=abs)
    assert np.all(abs(got - ref) <= bound * terms)


@pytest.mark.parametrize("nodes,Nq,cq", [("gauss", 3, 5), ("gauss", 5, 5), ("gauss", 3, 3), ("gauss", 7, 7),
                                         ("gauss", 8, 12), ("lobatto", 2, 3), ("lobatto", 3, 5), ("lobatto", 8, 12)])
@pytest.mark.parametrize("kind", ["metric spike", "metric plane", "metric ends", "velocity spike", "boundary layer"])
def test_cubature_component_by_component(nb, O, dev, nodes, Nq, cq, kind):
    check(nb, O, dev, nodes, Nq, cq, 6, kind, 1.2e-9)


@pytest.mark.parametrize("Nq", [2, 3, 4, 8, 12])
@pytest.mark.parametrize("kind", ["velocity spike", "boundary layer", "metric spike", "uniform"])
def test_own_nodes_component_by_component(nb, O, dev, Nq, kind):
    check(nb, O, dev, "own", Nq, Nq, 2 if Nq == 12 else 40, kind, 1.3e-11)


@pytest.mark.parametrize("Nq,E", [(2, 5000), (5, 1000), (8, 400)])
def test_own_nodes_whole_and_in_parts(nb, O, dev, Nq, E):
    """More elements than resident CTAs, one of them without a fixed-point form: the others have the bits
    of a call of their own."""
    x = O.gll(Nq - 1)[0]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a).ravel()).to(dev)  # noqa: E731
    rng = np.random.default_rng(Nq)
    U = rng.uniform(-1, 1, (3, E, Nq ** 3))
    U[1, E // 2, 1] = np.inf
    g, vg = (rng.uniform(0.5, 1.5, (E, NVGEO, Nq ** 3)) for _ in range(2))
    D, I = t(O.dmatrix(x)), t(np.eye(Nq))

    def run(a, b):
        NU = torch.full((3 * (b - a) * Nq ** 3,), 5.0, dtype=torch.float64, device=dev)
        nb.adv_cubature(Nq, Nq, b - a, t(vg[a:b]), t(g[a:b]), D, I, (b - a) * Nq ** 3, t(U[:, a:b]), NU)
        return NU.cpu().numpy().reshape(3, b - a, -1)

    whole, e = run(0, E), E // 2
    assert not np.isfinite(whole[:, e]).all() and np.isfinite(np.delete(whole, e, 1)).all()
    for a, b in ((0, 1), (7, 9), (e + 1, E)):
        assert np.array_equal(whole[:, a:b], run(a, b))
