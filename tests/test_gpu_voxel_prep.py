"""gbsimp_voxel_prep at the edges of its kernels: extents of one, of a row more or less than a tile of 32,
wide bands, steep and reversed logistics, and values that a double-float sum cannot hold."""
import numpy as np
import pytest
import torch

from genpipeline_gb300.engine import get_engine
from oracle import voxel_oracle as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma,sharp", [(0.0, 15.0), (0.5, 15.0), (1.5, -40.0), (0.7, 400.0)])
@pytest.mark.parametrize("shape,out", [((1, 1, 1), (1, 1, 1)), ((2, 31, 33), (2, 16, 17)), ((7, 9, 64), (7, 5, 33)),
                                       ((5, 64, 65), (9, 32, 32)), ((17, 3, 130), (9, 2, 65))])
def test_matches_fp64(shape, out, sigma, sharp):
    vol = np.random.default_rng(7).random((3, *shape), dtype=np.float32)
    got = get_engine().voxel_prep(torch.from_numpy(vol).cuda(), out, sigma, sharp).cpu().numpy()
    # two FP32 roundings of values below 1 on the way, through a slope of sharpness / 4, and the last one
    tol = 2 * 2.0 ** -25 * abs(sharp) / 4 + 2.0 ** -24
    for b in range(3):
        with np.errstate(over="ignore"):
            assert np.abs(got[b] - V.voxel_prep(vol[b], out, sigma, sharp)).max() <= tol


def test_values_outside_the_range_of_a_pair():
    v = np.full((3, 3, 3), 0.25, dtype=np.float32)
    v[1, 1, 1] = np.inf  # under a weight of zero everywhere: never seen
    got = get_engine().voxel_prep(torch.from_numpy(v).cuda(), (2, 2, 2), 0.0, 4.0).cpu().numpy()
    np.testing.assert_allclose(got, 1 / (1 + np.exp(1.0)), rtol=2.0 ** -23)
    v = np.array([np.inf, -np.inf, np.nan, 3e38, -3e38, 1e-40, 0.0, -0.0, 1e-35], dtype=np.float32).reshape(1, 1, 9)
    got = get_engine().voxel_prep(torch.from_numpy(v).cuda(), (1, 1, 9), 0.0, 2.0).cpu().numpy().reshape(-1)
    with np.errstate(over="ignore", invalid="ignore"):
        want = 1 / (1 + np.exp(-2.0 * (v.reshape(-1).astype(np.float64) - 0.5)))
    np.testing.assert_allclose(got, want, rtol=2.0 ** -23)
    one = np.zeros((4, 4, 4), dtype=np.float32)
    one[0, 0, 0] = np.nan
    got = get_engine().voxel_prep(torch.from_numpy(one).cuda(), (4, 4, 4), 0.3, 15.0).cpu().numpy()
    assert np.isnan(got).sum() == 8 and np.isnan(got[:2, :2, :2]).all()  # radius one, mirrored at the border


@pytest.mark.parametrize("void", [1e-29, 1e-32, 1e-38, 1e-44])
@pytest.mark.parametrize("shape,out", [((5, 33, 64), (3, 17, 32)), ((40, 3, 65), (20, 2, 33))])
def test_a_void_of_small_values(shape, out, void):
    """Solids in a void at the low end of the FP32 range, as a steep decoder leaves it."""
    rng = np.random.default_rng(3)
    vol = np.where(rng.random(shape) < 0.5, rng.random(shape), void * rng.random(shape)).astype(np.float32)
    vol[: shape[0] // 2] = void
    got = get_engine().voxel_prep(torch.from_numpy(vol).cuda(), out).cpu().numpy()
    # as above: two FP32 roundings through a slope of 15 / 4, and the last one
    assert np.abs(got - V.voxel_prep(vol, out)).max() <= 2 * 2.0 ** -25 * 15 / 4 + 2.0 ** -24
