"""The on-chip PCG (csrc/pcg_chip.cu) at the edges of its boxes: one element, rows of one and of 33
elements, uneven cuts, one to six places per thread, the largest cube, and a grid one step past it
that streams instead; straight through and paused every few iterations."""
import threading

import numpy as np
import pytest
import torch

from genpipeline_gb300 import _lib as L
from genpipeline_gb300 import bcs
from genpipeline_gb300.batch import BatchFEM, FEMDesign
from genpipeline_gb300.engine import get_engine, n_dof, n_elem
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pause", [0, 7])
@pytest.mark.parametrize("grid", [(1, 1, 1), (3, 2, 33), (5, 1, 64), (16, 8, 8), (33, 17, 9), (7, 41, 30), (48, 48, 48),
                                  (64, 64, 64), (66, 66, 66)])
def test_on_chip_solution_meets_its_tolerance(grid, pause):
    eng = get_engine()
    f, fixed = bcs.LOAD_CASES["cantilever"](*grid)
    x = np.random.default_rng(5).uniform(0.2, 1.0, n_elem(grid)).astype(np.float32)
    if pause:
        d = FEMDesign(grid, x, f, fixed)
        BatchFEM(eng, L.make_law("modified", 3.0), rtol=1e-8, round_iters=pause).solve_all([d])
        u, st = d.du, d.stats
    else:
        u = torch.zeros(n_dof(grid), dtype=torch.float64, device="cuda")
        st = eng.solve(grid, L.make_law("modified", 3.0), torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(),
                       torch.from_numpy(bcs.node_mask(*grid, fixed)).cuda(), u, rtol=1e-8)
    assert st["status"] == L.GBS_OK and st["relres"] <= 1e-8, st
    dof = bcs.dof_mask(*grid, fixed)
    E = O.moduli(x.astype(np.float64), O.Material("modified", penal=3.0, emin=1e-9))
    r = f - O.apply(grid, O.ke_quadrature(), E, u.cpu().numpy(), dof)
    free = np.asarray(dof) == 0
    # the residual that stopped the solve carries 2^-46 of the displacements, up to the squared length
    # of the grid above the load: 6e-11
    assert np.linalg.norm(r[free]) <= (1e-8 + 1e-10) * np.linalg.norm(f[free])


def test_solves_on_several_threads_and_streams():
    """Cooperative launches from four threads, each on its own stream: the same displacements as alone."""
    eng, law = get_engine(), L.make_law("modified", 3.0)
    grids = [(32, 32, 32), (48, 20, 20), (64, 64, 40), (16, 8, 8)]
    cases = []
    for g in grids:
        f, fixed = bcs.LOAD_CASES["cantilever"](*g)
        x = np.random.default_rng(8).uniform(0.2, 1.0, n_elem(g)).astype(np.float32)
        cases.append((g, torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(),
                      torch.from_numpy(bcs.node_mask(*g, fixed)).cuda()))
    alone = []
    for k, (g, x, f, m) in enumerate(cases):
        u = torch.zeros_like(f)
        assert eng.solve(g, law, x, f, m, u, key=f"alone{k}")["status"] == L.GBS_OK
        alone.append(u)
    torch.cuda.synchronize()
    got, errors = [None] * 4, []

    def work(k):
        try:
            g, x, f, m = cases[k]
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(6):
                    u = torch.zeros_like(f)
                    st = eng.solve(g, law, x, f, m, u, key=f"thread{k}")
                    assert st["status"] == L.GBS_OK, st
                torch.cuda.current_stream().synchronize()
                got[k] = u
        except BaseException as e:  # reported below: a thread's exception is lost otherwise
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, got):
        assert torch.equal(a, b)
