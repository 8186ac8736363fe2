"""The advection operator's fixed-point contractions (csrc/adv_fx.cuh) where a zero of a matrix
meets values that are far apart along a line, against extended precision (np.longdouble) on the same
operands, component by component.

A contraction is off by at most (cq + 2) 2^-54 of max|M| max|v| of its row and line.  Lines in
which one value is more than 2^(far + 1) above all others go to the FP64 sums where a row has terms
below 2^-9 max|M| max|v|, and entries of these
matrices beside their zeros are within 2^r of their row's largest: cq = 3 (far 10, r 3)
5 2^-54 2^14 = 4.5e-12 of the terms, cq = 12 (6, 10.2) 14 2^-54 2^17.2 = 1.2e-10, the others less; nine
contractions stay below 1.2e-9.  Where all is done in FP64 sums (66 roundings), 1e-14."""
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
    xc = O.gauss(cq - 1)[0] if nodes == "gauss" else xg
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


@pytest.mark.parametrize("Nq,cq", [(3, 5), (5, 5), (3, 3), (7, 7), (8, 12)])
@pytest.mark.parametrize("kind", ["metric spike", "metric plane", "velocity spike", "boundary layer"])
def test_gauss_cubature_component_by_component(nb, O, dev, Nq, cq, kind):
    check(nb, O, dev, "gauss", Nq, cq, 6, kind, 1.2e-9)


@pytest.mark.parametrize("Nq", [3, 4, 8])
@pytest.mark.parametrize("kind", ["velocity spike", "boundary layer", "metric spike"])
def test_collocated_cubature_component_by_component(nb, O, dev, Nq, kind):
    check(nb, O, dev, "own", Nq, Nq, 4, kind, 1e-14)
