"""Calls that find the on-chip PCG's cooperative launch refused (a context that may use fewer SMs than the
device has, say; here the library is told to take it so) go on in the streaming forms."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.engine import Engine, n_dof, n_elem

pytestmark = pytest.mark.gpu
LAW = L.make_law("modified", 3.0)


def _engine(value=1):
    eng = Engine()
    L.check(eng.lib.gbsimp_set_diagnostic(eng.ctx, L.DIAG_CHIP, value))
    return eng


def _case(grid):
    f, fixed = bcs.LOAD_CASES["cantilever"](*grid)
    x = np.random.default_rng(5).uniform(0.2, 1.0, n_elem(grid)).astype(np.float32)
    return torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), torch.from_numpy(bcs.node_mask(*grid, fixed)).cuda()


@pytest.mark.parametrize("profile", [False, True])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("residual_fp64", [False, True])
@pytest.mark.parametrize("grid", [(16, 8, 8), (33, 17, 9)])
def test_solve(grid, residual_fp64, fused, profile):
    x, f, mask = _case(grid)
    u, v = torch.zeros(n_dof(grid), dtype=torch.float64, device="cuda"), torch.zeros(n_dof(grid), dtype=torch.float64, device="cuda")
    kw = dict(fused=fused, residual_fp64=residual_fp64, profile=profile)
    st = _engine().solve(grid, LAW, x, f, mask, u, **kw)
    assert st["status"] == L.GBS_OK and st["relres"] <= 1e-8, st
    # the same as in a context where the chip holds nothing
    want = _engine(0).solve(grid, LAW, x, f, mask, v, **kw)
    assert st["iterations"] == want["iterations"] and torch.equal(u, v)


def test_pcg_from_a_guess_and_the_timing_call():
    grid = (16, 8, 8)
    x, f, mask = _case(grid)
    b = f.float()
    u0 = torch.randn_like(b)
    u, v = u0.clone(), u0.clone()
    st = _engine().pcg(grid, LAW, x, b, mask, u, rtol=1e-4)
    want = _engine(0).pcg(grid, LAW, x, b, mask, v, rtol=1e-4)
    assert st["status"] == L.GBS_OK and st["iterations"] == want["iterations"] and torch.equal(u, v)
    assert 0 < _engine().time_pcg_apply(grid, LAW, x, mask, reps=5) < 1e-3
