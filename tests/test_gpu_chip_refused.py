"""Calls that find the on-chip PCG's cooperative launch refused (a context that may use fewer SMs than the
device has, say; here the library is told to take it so) go on in the streaming forms."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import Engine, n_dof, n_elem
from oracle import oracle as O

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


def _designs():
    out = []
    for g in [(16, 8, 8), (20, 20, 20), (30, 11, 40)]:
        f, fixed = bcs.LOAD_CASES["cantilever"](*g)
        out.append(FEMDesign(g, np.random.default_rng(8).uniform(0.2, 1.0, n_elem(g)).astype(np.float32), f, fixed))
    return out


def _check(d):
    assert d.stats["status"] == L.GBS_OK and d.stats["relres"] <= 1e-8, d.stats
    dof = bcs.dof_mask(*d.grid, d.fixed_dofs)
    E = O.moduli(d.x.astype(np.float64), O.Material("modified", penal=3.0, emin=1e-9))
    r = d.f - O.apply(d.grid, O.ke_quadrature(), E, d.du.cpu().numpy(), dof)
    free = np.asarray(dof) == 0
    # the residual that stopped the solve carries 2^-46 of the displacements, at most the grid's squared
    # length above the load
    assert np.linalg.norm(r[free]) <= (1e-8 + 1e-10) * np.linalg.norm(d.f[free])


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("pause", [0, 40])
def test_batch(fused, pause):
    designs = _designs()
    BatchFEM(_engine(), LAW, fused=fused, round_iters=pause).solve_all(designs)
    for d in designs:
        _check(d)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("before,after", [(-1, 1), (-1, 0), (0, -1)])
def test_a_paused_batch_goes_on_when_the_chip_comes_or_goes(before, after, fused):
    """Solves paused in one form are not resumed in another: each ends at its tolerance."""
    eng, designs = _engine(before), _designs()
    b = BatchFEM(eng, LAW, fused=fused, round_iters=40)
    for d in designs:
        b.add(d)
    for k in range(4000):
        if k == 3:
            L.check(eng.lib.gbsimp_set_diagnostic(eng.ctx, L.DIAG_CHIP, after))
        b.round()
        if not b.items:
            break
    for d in designs:
        _check(d)
