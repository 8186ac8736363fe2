"""Every kernel of a captured iteration is prepared by a launch before the capture: a fresh process,
whose first solve is the one in question."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOLVE = """
import os, sys
sys.path.insert(0, {root!r})
import torch
import nekbench_gb300 as nb
bp = nb.BP({N}, {n}, Nfields={nf}, perturb=0.1)
f = torch.rand({nf} * bp.Nlocal, dtype=torch.float64, device="cuda") - 0.5
bp.ogs.gather_scatter_many(f, {nf}, bp.Nlocal)
lam = torch.ones(2 * bp.Nlocal, dtype=torch.float64, device="cuda")
net = nb.Net.load(os.path.join(os.path.dirname(nb.__file__), "weights", "precond_n7_c16.bin")) if {learned} else None
kw = dict(precond=nb.PRECOND_LEARNED, net=net, fcg_window={learned}) if {learned} else {{}}
st = bp.pcg(lam, f, torch.zeros_like(f), 1e-6, 500, solver=nb.{solver}, inner_precision=nb.{inner}, **kw)
assert st["status"] == 0, st
print("prepared in a capture:", nb.lib().nekb_captured_opt_ins())
"""


@pytest.mark.parametrize("N,n,nf,solver,inner,learned", [
    (3, 3, 1, "SOLVER_FP64", "FP32", 0), (3, 3, 1, "SOLVER_FP64_SPLIT", "FP32", 0), (3, 3, 1, "SOLVER_MIXED", "FP32", 0),
    (9, 2, 1, "SOLVER_MIXED", "FP32", 0), (9, 2, 3, "SOLVER_MIXED", "FP32", 0), (7, 4, 1, "SOLVER_MIXED", "BF16", 0),
    (7, 4, 1, "SOLVER_MIXED", "FP32_TRILINEAR", 0), (7, 11, 1, "SOLVER_MIXED", "FP32", 0), (7, 4, 1, "SOLVER_MIXED", "FP32", 5),
    (7, 4, 1, "SOLVER_MIXED", "FP32", 1)])
def test_no_kernel_is_prepared_inside_a_capture(nb, dev, N, n, nf, solver, inner, learned):
    code = SOLVE.format(root=ROOT, N=N, n=n, nf=nf, solver=solver, inner=inner, learned=learned)
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    assert p.stdout.strip().endswith("prepared in a capture: 0"), p.stdout
