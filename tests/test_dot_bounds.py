"""Arrays shorter than what the dot kernels go through are refused before anything is launched:
for several fields the block kernel reads the weights per field, like x and y."""
import pytest
import torch

import nekbench_gb300 as nb


@pytest.mark.parametrize("t,n,fits", [(torch.zeros(8), 8, True), (torch.zeros(8), 9, False),
                                      (torch.zeros(8)[2:], 6, True), (torch.zeros(8)[2:], 7, False),
                                      (torch.zeros(8)[2:4], 6, True),  # a view: what lies behind it counts
                                      (torch.zeros(1).expand(8), 8, False), (torch.zeros(4, 4)[:, 0], 16, True),
                                      (4096, 100, True)])
def test_entries_held(t, n, fits):
    if fits:
        nb._require_entries(t=(t, n))
    else:
        with pytest.raises(nb.NekbError, match="are needed"):
            nb._require_entries(t=(t, n))


@pytest.mark.gpu
@pytest.mark.parametrize("short", ["w", "x", "y", "wxy"])
def test_short_arrays_are_refused(nb, O, dev, short):
    N, off, NF = 1000, 1003, 3
    a = {k: torch.rand(off * NF, dtype=torch.float64, device=dev) for k in "wxy"}
    a["wxy"] = torch.full((4,), 7.0, dtype=torch.float64, device=dev)
    kernel = nb.load_dot_kernel("weightedBlockInnerProduct2", 256, NF)
    kernel(N, off, *a.values())
    assert (a["wxy"].cpu().numpy() == O.dot_partials(2, *(a[k].cpu().numpy() for k in "wxy"), N=N, Nfields=NF,
                                                     offset=off, block_size=256)).all()
    a[short] = a[short][:3].clone() if short == "wxy" else a[short][:N].clone()
    a["wxy"].fill_(7.0)
    with pytest.raises(nb.NekbError):
        kernel(N, off, *a.values())
    assert (a["wxy"] == 7.0).all()
