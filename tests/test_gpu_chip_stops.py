"""Ends of an on-chip PCG (csrc/pcg_chip.cu) other than convergence."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import Engine, get_engine, n_dof, n_elem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(4, 3, 2), (32, 8, 8), (64, 64, 64)])
def test_a_zero_load_gives_zero_whatever_the_guess(grid):
    """D b = 0 ends the solve at its setup: the answer is zero, not the guess it started from."""
    _, fixed = bcs.LOAD_CASES["cantilever"](*grid)
    mask = torch.from_numpy(bcs.node_mask(*grid, fixed)).cuda()
    b = torch.zeros(n_dof(grid), device="cuda")
    b[bcs.dof_mask(*grid, fixed).astype(bool)] = 1.0  # on clamped DOFs only
    u = torch.ones_like(b)
    st = get_engine().pcg(grid, L.make_law("modified", 3.0), torch.ones(n_elem(grid), device="cuda"), b, mask, u)
    assert st["status"] == L.GBS_OK and st["iterations"] == 0
    assert not u.any()


def _late(block=0):
    """An engine of its own whose waits for other blocks run out (block b > 0: only reports so at its end)."""
    eng = Engine()
    L.check(eng.lib.gbsimp_set_diagnostic(eng.ctx, L.DIAG_TIMEOUT, block))
    return eng


def _case(grid):
    f, fixed = bcs.LOAD_CASES["cantilever"](*grid)
    x = np.random.default_rng(5).uniform(0.2, 1.0, n_elem(grid)).astype(np.float32)
    return (torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), torch.from_numpy(bcs.node_mask(*grid, fixed)).cuda(),
            FEMDesign(grid, x, f, fixed))


@pytest.mark.parametrize("residual_fp64", [False, True])
@pytest.mark.parametrize("grid", [(16, 8, 8), (32, 32, 32), (64, 64, 64)])
def test_a_timed_out_solve_leaves_u_and_says_so(grid, residual_fp64):
    law, (x, f, mask, _) = L.make_law("modified", 3.0), _case(grid)
    eng = _late()
    eng.workspace("solve", int(eng.lib.gbsimp_solve_ws_bytes(*grid))).fill_(0xFF)  # NaN everywhere
    u0 = torch.randn(n_dof(grid), dtype=torch.float64, device="cuda")
    u0[torch.from_numpy(bcs.dof_mask(*grid, bcs.LOAD_CASES["cantilever"](*grid)[1])).cuda().bool()] = 0.0
    u = u0.clone()
    st = eng.solve(grid, law, x, f, mask, u, residual_fp64=residual_fp64)
    assert st["status"] == L.GBS_ETIMEOUT, st
    assert torch.equal(u, u0)
    # the context and the workspace work on
    L.check(eng.lib.gbsimp_set_diagnostic(eng.ctx, L.DIAG_TIMEOUT, -1))
    st = eng.solve(grid, law, x, f, mask, u, residual_fp64=residual_fp64)
    assert st["status"] == L.GBS_OK and st["relres"] <= 1e-8, st


def test_a_timed_out_design_of_a_batch_leaves_u_and_says_so():
    designs = [_case(g)[3] for g in [(20, 20, 20), (28, 31, 30), (32, 32, 32)]]  # more than one block holds
    BatchFEM(_late()).solve_all(designs)
    for d in designs:
        assert d.stats["status"] == L.GBS_ETIMEOUT and not d.du.any()


@pytest.mark.parametrize("block", [0, 1, 7])
def test_a_block_that_gives_up_last_is_not_overruled(block):
    """rtol above 1 ends a solve at its first sums, so that the first block leaves the loop as usual while
    another one's wait has run out: the solve's status is the timeout all the same."""
    grid = (32, 32, 32)
    x, f, mask, _ = _case(grid)
    law = L.make_law("modified", 3.0)
    for _ in range(5):
        u = torch.zeros(n_dof(grid), dtype=torch.float64, device="cuda")
        st = _late(block).solve(grid, law, x, f, mask, u, rtol=1e-8, inner_rtol=2.0)
        assert st["status"] == L.GBS_ETIMEOUT and not u.any(), st


@pytest.mark.parametrize("grid", [(61, 37, 23), (128, 64, 64)])
def test_a_timed_out_oc_update_says_so(grid):
    eng, n = _late(), n_elem(grid)
    x, dc = torch.full((n,), 0.4, device="cuda"), -torch.rand(n, device="cuda")
    eng.oc(grid, 1.5, 0.3, x, dc)
    with pytest.raises(L.GbsimpError) as e:
        eng.oc_result()
    assert e.value.code == L.GBS_ETIMEOUT
    L.check(eng.lib.gbsimp_set_diagnostic(eng.ctx, L.DIAG_TIMEOUT, -1))
    want = get_engine().oc(grid, 1.5, 0.3, x, dc)
    got = eng.oc(grid, 1.5, 0.3, x, dc)
    assert eng.oc_result()[1] > 0 and all(torch.equal(a, b) for a, b in zip(got, want))
