"""Which form a batch's inner solves take: on the chip side by side, or together in persistent launches where
the chip would hold them one after the other for longer; the displacements meet the tolerance in both."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import n_elem
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KERNEL = {"chip": "pcg_chip_kernel", "persistent": "pcg_fused_kernel", "graph": "apply_modal_kernel"}
PAUSED = {1: "persistent", 2: "graph", 3: "chip"}  # stats.inner_active


def _designs(sizes):
    out = []
    for k, n in enumerate(sizes):
        g = (n, n, n) if np.isscalar(n) else n
        f, fixed = bcs.LOAD_CASES["cantilever"](*g)
        out.append(FEMDesign(g, np.random.default_rng(k).uniform(0.3, 1.0, n_elem(g)).astype(np.float32), f, fixed))
    return out


def _kernels(run):
    """The names of the kernels that run() launches."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    return {e.name for e in prof.events()}


@pytest.fixture(scope="module", autouse=True)
def tracing():
    """A process's first profile may come back empty."""
    for _ in range(5):
        if _kernels(lambda: torch.zeros(1 << 20, device="cuda").add_(1)):
            return
    pytest.skip("no kernel names from the profiler here")


@pytest.mark.parametrize("sizes,fused,form,paused", [
    ((57,) * 2, True, "chip", "chip"), ((57,) * 5, True, "persistent", "chip"), ((57,) * 5, False, "chip", "chip"),
    ((64,) * 4, True, "chip", "chip"), ((64,) * 6, True, "persistent", "chip"), ((32,) * 20, True, "chip", "chip"),
    ((8,) * 30, True, "chip", "chip"), ((67, 67), True, "persistent", "persistent"), ((67, 67), False, "graph", "graph")])
def test_form_and_residual(sizes, fused, form, paused):
    # rounds of whole inner solves
    designs = _designs(sizes)
    b = BatchFEM(fused=fused)
    for d in designs:
        b.add(d)
    names = _kernels(b.round)
    assert {f for f, k in KERNEL.items() if any(k in n for n in names)} == {form}
    while b.items:
        b.round()
    _check(designs)
    # rounds of a budget
    designs = _designs(sizes)
    b = BatchFEM(fused=fused, round_iters=24)
    for d in designs:
        b.add(d)
    b.round()
    assert {PAUSED[d._item.stats.inner_active] for d in designs} == {paused}
    b.opts.check_every = 0
    while b.items:
        b.round()
    _check(designs)


def _check(designs):
    for d in designs[:3]:
        assert d.stats["status"] == L.GBS_OK and d.stats["relres"] <= 1e-8, d.stats
        dof = bcs.dof_mask(*d.grid, d.fixed_dofs)
        E = O.moduli(d.x.astype(np.float64), O.Material("modified", penal=3.0, emin=1e-9))
        r = d.f - O.apply(d.grid, O.ke_quadrature(), E, d.du.cpu().numpy(), dof)
        free = np.asarray(dof) == 0
        # the residual that stopped the solve carries 2^-46 of the displacements, at most the grid's squared
        # length above the load
        assert np.linalg.norm(r[free]) <= (1e-8 + 1e-10) * np.linalg.norm(d.f[free])
