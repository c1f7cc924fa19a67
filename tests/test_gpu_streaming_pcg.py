"""The streaming forms of the PCG (graph loop and persistent kernel), which every grid that the chip does not
hold runs in: here on small grids, in a context where the chip holds none, with the rules, tolerances and
shapes of the tests that the on-chip form now answers elsewhere."""
import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300 import designs as D
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import Engine, n_dof, n_elem
from oracle import oracle as O

pytestmark = pytest.mark.gpu
LAW = L.make_law("modified", 3.0)
MAT = O.Material("modified", 3.0, emin=1e-9)
PERSISTENT, GRAPH = 1, 2  # stats.inner_active of a paused solve


@pytest.fixture(scope="module")
def eng():
    e = Engine()
    L.check(e.lib.gbsimp_set_diagnostic(e.ctx, L.DIAG_CHIP, 0))
    return e


def _problem(grid, case="cantilever", seed=5):
    f, fixed = bcs.LOAD_CASES[case](*grid)
    x = np.random.default_rng(seed).uniform(0.05, 1.0, n_elem(grid)).astype(np.float32)
    return torch.from_numpy(f).cuda(), torch.from_numpy(bcs.node_mask(*grid, fixed)).cuda(), torch.from_numpy(x).cuda(), f, fixed


def _zeros(grid):
    return torch.zeros(n_dof(grid), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("grid,case", [((24, 12, 12), "top_patch"), ((64, 32, 32), "cantilever"),
                                       ((40, 20, 100), "edge_line")])
def test_persistent_matches_graph_loop_and_the_chip(eng, grid, case):
    """Three forms, one solution: displacements to the solve's tolerance, iteration counts within 12 % (the
    forms round differently, and where an inner solve stops depends on that)."""
    f, m, x, _, _ = _problem(grid, case)
    out = []
    for e, fused in ((eng, False), (eng, True), (Engine(), False)):
        u = _zeros(grid)
        before = e.lib.gbsimp_launch_count()
        st = e.solve(grid, LAW, x, f, m, u, rtol=1e-8, fused=fused)
        launches = e.lib.gbsimp_launch_count() - before
        assert st["status"] == L.GBS_OK and st["relres"] <= 1e-8, st
        # the graph loop launches once per iteration, the others once per inner solve
        assert (launches >= st["iterations"]) == (e is eng and not fused), (launches, st)
        out.append((u, st["iterations"]))
    for u, its in out[1:]:
        assert float((u - out[0][0]).abs().max()) <= 1e-6 * float(out[0][0].abs().max())
        assert abs(its - out[0][1]) <= max(5, 0.12 * out[0][1])


@pytest.mark.parametrize("fused", [False, True])
def test_deterministic(eng, fused):
    grid = (32, 16, 16)
    f, m, x, _, _ = _problem(grid)
    got = []
    for _ in range(3):
        u = _zeros(grid)
        eng.solve(grid, LAW, x, f, m, u, rtol=1e-8, fused=fused)
        got.append(u)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("fused", [False, True])
def test_stop_rules_of_the_start(eng, fused):
    """A cap of 5 ends the inner solve after 5 iterations; a tolerance above 1 is met by x0 = 0."""
    grid = (12, 6, 6)
    f, m, x, _, _ = _problem(grid)
    u = _zeros(grid)
    st = eng.solve(grid, LAW, x, f, m, u, max_iter=5, fused=fused)
    assert st["status"] == L.GBS_ENOTCONV and st["iterations"] == 5, st
    assert 0.0 < st["relres"] < 1.0 and torch.isfinite(u).all()
    u.zero_()
    st = eng.solve(grid, LAW, x, f, m, u, inner_rtol=2.0, max_outer=3, fused=fused)
    assert st["status"] == L.GBS_ENOTCONV and st["iterations"] == 0 and not u.any(), st


@pytest.mark.parametrize("fused", [False, True])
def test_pcg_cap_zero_load_and_nan(eng, fused):
    grid = (8, 4, 4)
    f, m, x, _, fixed = _problem(grid)
    b = f.float()
    u = torch.zeros_like(b)
    st = eng.pcg(grid, LAW, x, b, m, u, rtol=1e-12, max_iter=3, fused=fused)
    assert st["status"] == L.GBS_ENOTCONV and st["iterations"] == 3
    u.fill_(1.0)
    st = eng.pcg(grid, LAW, x, torch.zeros_like(b), m, u, fused=fused)
    assert st["status"] == L.GBS_OK and st["iterations"] == 0 and not u.any()
    x[5] = float("nan")
    u.zero_()
    st = eng.pcg(grid, LAW, x, b, m, u, rtol=1e-6, max_iter=50, fused=fused)
    assert st["status"] in (L.GBS_ENONFINITE, L.GBS_EBREAKDOWN)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("grid", [(8, 4, 167), (8, 4, 200), (3, 2, 446)])
def test_tall_z_against_oracle(eng, grid, fused):
    f, m, x, fh, fixed = _problem(grid)
    uref, _, _ = O.pcg(grid, O.ke_quadrature(), O.moduli(x.cpu().numpy().astype(np.float64), MAT), fh,
                       bcs.dof_mask(*grid, fixed), tol=1e-13)
    u = _zeros(grid)
    st = eng.solve(grid, LAW, x, f, m, u, rtol=1e-8, fused=fused)
    assert st["status"] == L.GBS_OK and st["relres"] <= 1e-8, st
    ug = u.cpu().numpy()
    assert float(fh @ ug) == pytest.approx(float(fh @ uref), rel=1e-6)
    np.testing.assert_allclose(ug, uref, rtol=0, atol=1e-5 * np.abs(uref).max())


def _designs():
    out = []
    for k, (grid, load) in enumerate([((24, 24, 24), "cantilever"), ((32, 32, 32), "top_patch"),
                                      ((40, 20, 20), "cantilever"), ((16, 16, 16), "torsion"),
                                      ((48, 24, 12), "cantilever")]):
        f, fixed = bcs.cantilever_tip(*grid) if load == "cantilever" else D.load_case(load, grid[0])
        out.append(FEMDesign(grid, D.grf_density(grid, 100 + k), f, fixed))
    return out


@pytest.mark.parametrize("fused,round_iters,share,group", [(True, 0, 0, 0), (False, 0, 0, 0), (True, 7, 0, 0),
                                                           (False, 30, 0, 0), (True, 0, 1, 0), (True, 13, 1, 2)])
def test_batch_equals_the_chips(eng, fused, round_iters, share, group):
    """Designs sharing persistent launches or each in its graph loop, whole inner solves or paused every few
    iterations, SM shares, launches of two: the displacements that the chip gives."""
    want = {d.grid: d for d in BatchFEM(Engine()).solve_all(_designs())}
    b = BatchFEM(eng, fused=fused, round_iters=round_iters)
    b.opts.batch_share, b.opts.batch_group = share, group
    designs = _designs()
    for d in designs:
        b.add(d)
    seen = set()
    while b.items:
        b.round()
        seen |= {d._item.stats.inner_active for d in b.items}
    assert seen - {0} == (set() if round_iters == 0 else {PERSISTENT if fused else GRAPH})
    for d in designs:
        w = want[d.grid]
        assert d.stats["status"] == L.GBS_OK and d.stats["relres"] <= 1e-8, d.stats
        # both are solved to 1e-8 of the load: 1e-6 of the largest displacement
        assert float((d.du - w.du).abs().max()) <= 1e-6 * float(w.du.abs().max())


@pytest.mark.parametrize("fused", [False, True])
def test_solves_past_the_chip_need_no_switch(fused):
    """The first cube that the chip does not hold, in an ordinary context."""
    eng, grid = Engine(), (67, 67, 67)
    f, m, x, fh, fixed = _problem(grid)
    x.clamp_(min=0.3)
    u = _zeros(grid)
    st = eng.solve(grid, LAW, x, f, m, u, rtol=1e-8, fused=fused)
    assert st["status"] == L.GBS_OK and st["relres"] <= 1e-8, st
    dof = bcs.dof_mask(*grid, fixed)
    r = fh - O.apply(grid, O.ke_quadrature(), O.moduli(x.cpu().numpy().astype(np.float64), MAT), u.cpu().numpy(), dof)
    free = np.asarray(dof) == 0
    # the residual that stopped the solve carries 2^-46 of the displacements, at most the grid's squared
    # length above the load
    assert np.linalg.norm(r[free]) <= (1e-8 + 1e-10) * np.linalg.norm(fh[free])
