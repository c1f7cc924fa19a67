"""The bare apply at the edges of its tiles and segments: one node plane per slab, odd numbers of planes, a
tile's last node, the tallest z, fixed DOFs, operands at any alignment, and values that may not spread."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300.engine import get_engine, n_dof, n_elem
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 1, 3), (3, 22, 20), (4, 23, 21), (7, 5, 446), (31, 90, 2), (152, 3, 3),
                                  (33, 40, 40)])
def test_apply_against_oracle(grid, masked):
    eng, rng = get_engine(), np.random.default_rng(2)
    x = rng.uniform(0.1, 1.0, n_elem(grid)).astype(np.float32)
    p = rng.standard_normal(n_dof(grid)).astype(np.float32)
    m = rng.integers(0, 8, n_dof(grid) // 3).astype(np.uint8) if masked else None
    dof = ((m[:, None] >> np.arange(3)) & 1).reshape(-1).astype(np.uint8) if masked else None
    buf = torch.empty(n_dof(grid) + 1, device="cuda")
    pd = buf[1:]  # four bytes off every wider alignment
    pd.copy_(torch.from_numpy(p))
    y = eng.apply(grid, L.make_law("modified", 3.0), torch.from_numpy(x).cuda(), pd,
                  torch.from_numpy(m).cuda() if masked else None).cpu().numpy()
    E = O.moduli(x.astype(np.float64), O.Material("modified", penal=3.0, emin=1e-9))
    want = O.apply(grid, O.ke_quadrature(), E, p.astype(np.float64), dof)
    # FP32 products of an element stiffness with entries up to 0.24 and 24 terms
    np.testing.assert_allclose(y, want, rtol=0, atol=2e-6 * np.abs(want).max())


def test_a_nan_stays_with_the_elements_that_touch_it():
    grid = (5, 6, 7)
    p = torch.zeros(6, 7, 8, 3, device="cuda")
    p[2, 3, 7, 1] = float("nan")
    y = get_engine().apply(grid, L.make_law("modified", 3.0), torch.ones(n_elem(grid), device="cuda"), p.reshape(-1))
    bad = torch.isnan(y.reshape(6, 7, 8, 3)).any(-1).cpu().numpy()
    want = np.zeros_like(bad)
    want[1:4, 2:5, 6:8] = True
    assert (bad == want).all()
