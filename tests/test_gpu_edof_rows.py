"""The kernels over an element -> DOF table at the edges of a block of rows, both index types, with indices
outside the vector (read as zero, not written) and energies that FP32 pairs do not hold."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import cuda_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_against_fp64(n, dtype):
    rng = np.random.default_rng(6)
    nd, R = 3 * n + 5, rng.standard_normal((24, 24))
    K = (R @ R.T).astype(np.float32)
    edof = rng.integers(-2, nd + 2, (n, 24))
    x, p = rng.uniform(0.1, 1, n).astype(np.float32), rng.standard_normal(nd).astype(np.float32)
    p[: nd // 2] *= 1e-18  # rows of tiny energies among them
    inside = (edof >= 0) & (edof < nd)
    pe = np.where(inside, p.astype(np.float64)[np.clip(edof, 0, nd - 1)], 0.0)
    ye = x.astype(np.float64)[:, None] ** 3 * (pe @ K.astype(np.float64))
    y = np.zeros(nd)
    np.add.at(y, edof[inside], ye[inside])
    t = lambda a, d=None: torch.as_tensor(a, device="cuda") if d is None else torch.as_tensor(a, device="cuda").to(d)
    args = (t(K), t(edof, dtype), 3.0, n, 1, 1)
    got = cuda_kernels.fused_spmv(t(x), t(p), *args).cpu().numpy()
    # 24 FP32 terms per row, up to a few dozen rows per DOF
    scale = np.abs(x[:, None] ** 3 * (np.abs(pe) @ np.abs(K))).max()
    np.testing.assert_allclose(got, y, rtol=0, atol=48 * 2.0 ** -24 * scale)
    dc = cuda_kernels.simp_sensitivity(t(x), t(p), *args).cpu().numpy()
    want = -3.0 * x.astype(np.float64) ** 2 * ((pe @ K) * pe).sum(1)
    bound = 3.0 * x.astype(np.float64) ** 2 * ((np.abs(pe) @ np.abs(K)) * np.abs(pe)).sum(1)
    assert (np.abs(dc - want) <= 30 * 2.0 ** -24 * bound + 2.0 ** -148).all()


def test_energies_outside_the_range_of_a_pair():
    K = torch.eye(24, device="cuda")
    edof = torch.arange(96, device="cuda").reshape(4, 24)
    u = torch.ones(96, device="cuda")
    u[:24], u[24:48], u[48] = 1e-21, 3e18, float("inf")
    dc = cuda_kernels.simp_sensitivity(torch.ones(4, device="cuda"), u, K, edof, 1.0, 4, 1, 1).cpu().numpy()
    np.testing.assert_allclose(dc[0], -24e-42, rtol=1e-3)
    np.testing.assert_allclose(dc[1], -24 * 9e36, rtol=1e-6)
    assert not np.isfinite(dc[2])
    np.testing.assert_allclose(dc[3], -24.0, rtol=1e-6)


@pytest.mark.parametrize("k", [-50, -45, -10, 15, 50])
def test_energies_scale_with_the_square_of_the_displacements(k):
    """A power of two in u is its square in the energy, to the last bit (energies from 1 to 1e4 here, so
    that FP32 holds both)."""
    rng = np.random.default_rng(2)
    n, nd = 300, 400
    R = rng.standard_normal((24, 24))
    K = torch.as_tensor((R @ R.T).astype(np.float32), device="cuda")
    edof = torch.as_tensor(rng.integers(0, nd, (n, 24)), device="cuda")
    x = torch.as_tensor(rng.uniform(0.5, 1, n).astype(np.float32), device="cuda")
    u = torch.as_tensor(rng.standard_normal(nd).astype(np.float32), device="cuda")
    want = cuda_kernels.simp_sensitivity(x, u, K, edof, 3.0, n, 1, 1)
    got = cuda_kernels.simp_sensitivity(x, u * 2.0 ** k, K, edof, 3.0, n, 1, 1) * 2.0 ** -k * 2.0 ** -k
    assert torch.equal(got, want)
