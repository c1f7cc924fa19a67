"""Ends of an on-chip PCG (csrc/pcg_chip.cu) other than convergence."""
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.engine import get_engine, n_dof, n_elem

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
