"""The tiled density filter at the edges of its tiles and for every reach of its stencil, against the FP64
oracle: both directions, the sums of weights, with and without them given, and preserved elements."""
import numpy as np
import pytest
import torch

from genpipeline_gb300.engine import get_engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rmin", [0.5, 1.0, 1.5, 2.3, 3.0, 4.2, 5.0, 6.0])
@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 3, 4), (5, 17, 33), (9, 40, 3), (65, 5, 8), (1, 2, 70), (40, 33, 32)])
def test_filter_against_oracle(grid, rmin):
    eng = get_engine()
    v = np.exp(np.random.default_rng(4).uniform(-12, 0, grid)).astype(np.float32)  # six decades
    d = torch.from_numpy(v).cuda().reshape(-1)
    hs = O.filter_hs(grid, rmin)
    got = eng.filter_hs(grid, rmin)
    # the weights', the products' and the sum's rounding; the transpose's division and hs come on top
    np.testing.assert_allclose(got.cpu().numpy(), hs.reshape(-1), rtol=3 * 2.0 ** -24)
    for transpose in (False, True):
        y = eng.filter(grid, rmin, d, hs=got, transpose=transpose).cpu().numpy()
        want = O.density_filter(grid, rmin, v.astype(np.float64).reshape(-1), hs=hs, transpose=transpose)
        np.testing.assert_allclose(y, np.asarray(want).reshape(-1), rtol=8 * 2.0 ** -24)
    np.testing.assert_allclose(eng.filter(grid, rmin, d).cpu().numpy(),
                               eng.filter(grid, rmin, d, hs=got).cpu().numpy(), rtol=2.0 ** -23)


@pytest.mark.parametrize("grid,rmin", [((48, 30, 33), 1.4), ((48, 30, 33), 1.5), ((32, 32, 32), 1.5), ((33, 33, 33), 1.5),
                                       ((32, 32, 32), 2.5), ((33, 33, 33), 2.5), ((4, 60, 15), 2.0), ((4, 60, 16), 2.0),
                                       ((1, 31, 3300), 2.5), ((1, 32, 3300), 2.5), ((1, 320, 320), 5.0), ((1, 320, 320), 5.5), ((1, 320, 320), 6.0),
                                       ((3300, 32, 1), 3.0), ((1, 1, 3000), 4.0), ((3000, 1, 1), 1.5)])
def test_both_forms_at_the_lines_between_them(grid, rmin):
    """Either side of each line of the choice between a tap at a time and tiles."""
    eng = get_engine()
    v = np.exp(np.random.default_rng(4).uniform(-12, 0, grid)).astype(np.float32)
    d = torch.from_numpy(v).cuda().reshape(-1)
    hs = O.filter_hs(grid, rmin)
    got = eng.filter_hs(grid, rmin)
    np.testing.assert_allclose(got.cpu().numpy(), hs.reshape(-1), rtol=3 * 2.0 ** -24)
    for transpose in (False, True):
        y = eng.filter(grid, rmin, d, hs=got, transpose=transpose).cpu().numpy()
        want = O.density_filter(grid, rmin, v.astype(np.float64).reshape(-1), hs=hs, transpose=transpose)
        np.testing.assert_allclose(y, np.asarray(want).reshape(-1), rtol=8 * 2.0 ** -24)
    np.testing.assert_allclose(eng.filter(grid, rmin, d).cpu().numpy(),
                               eng.filter(grid, rmin, d, hs=got).cpu().numpy(), rtol=2.0 ** -23)
