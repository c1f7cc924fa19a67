"""Which form a batch's inner solves take: on the chip side by side, or together in persistent launches where
the chip would hold them one after the other for longer; the displacements meet the tolerance in both."""
import numpy as np
import pytest

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import n_elem
from oracle import oracle as O

pytestmark = pytest.mark.gpu
PERSISTENT, GRAPH, CHIP = 1, 2, 3  # stats.inner_active of a paused solve


def _designs(sizes):
    out = []
    for k, n in enumerate(sizes):
        g = (n, n, n) if np.isscalar(n) else n
        f, fixed = bcs.LOAD_CASES["cantilever"](*g)
        out.append(FEMDesign(g, np.random.default_rng(k).uniform(0.3, 1.0, n_elem(g)).astype(np.float32), f, fixed))
    return out


@pytest.mark.parametrize("sizes,fused,form", [((57,) * 2, True, CHIP), ((57,) * 5, True, PERSISTENT),
                                              ((57,) * 5, False, CHIP), ((64,) * 4, True, CHIP),
                                              ((64,) * 6, True, PERSISTENT), ((32,) * 20, True, CHIP),
                                              ((8,) * 30, True, CHIP), ((67, 67), True, PERSISTENT),
                                              ((67, 67), False, GRAPH)])
def test_form_and_residual(sizes, fused, form):
    designs = _designs(sizes)
    b = BatchFEM(fused=fused, round_iters=24)
    for d in designs:
        b.add(d)
    b.round()
    assert {d._item.stats.inner_active for d in designs} == {form}
    b.opts.check_every = 0
    while b.items:
        b.round()
    for d in designs[:3]:
        assert d.stats["status"] == L.GBS_OK and d.stats["relres"] <= 1e-8, d.stats
        dof = bcs.dof_mask(*d.grid, d.fixed_dofs)
        E = O.moduli(d.x.astype(np.float64), O.Material("modified", penal=3.0, emin=1e-9))
        r = d.f - O.apply(d.grid, O.ke_quadrature(), E, d.du.cpu().numpy(), dof)
        free = np.asarray(dof) == 0
        # the residual that stopped the solve carries 2^-46 of the displacements, at most the grid's squared
        # length above the load
        assert np.linalg.norm(r[free]) <= (1e-8 + 1e-10) * np.linalg.norm(d.f[free])
