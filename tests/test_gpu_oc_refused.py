"""The OC update where its cooperative launch is refused: a launch per round, the same result."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300.engine import Engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["cpu", "gpu"])
@pytest.mark.parametrize("grid", [(8, 16, 16), (23, 17, 11), (96, 60, 40)])
def test_a_refused_launch_gives_the_oracles_update(grid, variant):
    eng = Engine()
    L.check(eng.lib.gbsimp_set_diagnostic(eng.ctx, L.DIAG_OC, 0))
    rng = np.random.default_rng(9)
    x = rng.uniform(0.0, 1, np.prod(grid)).astype(np.float32)
    dc = (-rng.gamma(2.0, 1.0, x.size)).astype(np.float32)
    pres = (rng.random(x.size) < 0.05).astype(np.uint8)
    vo, vl = (O.OC_CPU, L.OC_CPU) if variant == "cpu" else (O.OC_GPU, L.OC_GPU)
    xn_o, xp_o, it = O.oc(grid, 1.5, x, dc, 0.3, pres, variant=vo)
    xn, xp = eng.oc(grid, 1.5, 0.3, torch.from_numpy(x).cuda(), torch.from_numpy(dc).cuda(),
                    torch.from_numpy(pres).cuda(), vl)
    assert eng.oc_result()[1] == it
    # the multiplier is the oracle's interval: FP32 rounding of the update and of the filter is left
    np.testing.assert_allclose(xn.cpu().numpy(), xn_o, rtol=2e-6, atol=2e-7)
    np.testing.assert_allclose(xp.cpu().numpy(), xp_o, rtol=2e-6, atol=2e-7)
