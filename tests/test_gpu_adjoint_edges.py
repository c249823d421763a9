"""The transposed step at the edges of its work split, against the oracle's
FP64 adjoint: rows that end inside a column pair, one-row and one-plane
remainders of a z segment, slabs on some faces only, a design region that
touches the last column, two designs of different sizes in one sim, one
segment (recorded on the way) and several (re-run).  Tolerances are those of
test_gpu_adjoint.py: 1e-8 in FP64, 1e-3 in FP32, of the largest derivative."""
import numpy as np
import pytest

from oracle.oracle import OracleFields
from sim_juncs_gb300 import _abi
from sim_juncs_gb300.configs import AU, adjoint_case, junction_instance
from sim_juncs_gb300.fields import Fields
from sim_juncs_gb300.geometry import Box
from sim_juncs_gb300.spec import PML, Design, Grid, Objective, Region, Scene

pytestmark = pytest.mark.gpu

STEPS = 90


def case(nx, ny, nz, thickness, lo, dn, seed):
    inst = junction_instance(n=32, res=10.0, probe_components=("Ex",), dft=False)
    dx = inst.grid.dx
    inst.grid = Grid(nx, ny, nz, dx, inst.grid.dt)
    inst.pml = PML([[t * dx for t in pair] for pair in thickness])
    mid = [nx * dx / 2, ny * dx / 2, nz * dx / 2]
    inst.material = Scene([Region(Box((mid[0] - 0.45, mid[1] - 0.3, mid[2] - 0.2), (mid[0] + 0.1, mid[1] + 0.3, mid[2] + 0.1)),
                                  1.0, list(AU))])
    src = inst.sources[0]
    src.start_time, src.end_time = -9.0, 11.0
    src.lo, src.hi = (0.0, 0.0, mid[2] - 0.35), (nx * dx, ny * dx, mid[2] - 0.35)
    inst.probes = []
    eps = np.random.default_rng(seed).uniform(1.0, 4.0, size=(dn[2], dn[1], dn[0]))
    k = lo[2]
    cells = np.array([[lo[0], lo[1], k], [lo[0] + 1, lo[1], k], [nx - 1, ny - 1, nz // 2]])
    return inst, Design(lo, eps), Objective(cells, frequency=1 / 0.7, comps=(0, 1, 2))


GRIDS = {
    "odd": (33, 19, 17, [[4, 5], [3, 0], [0, 4]], (12, 8, 9), (5, 4, 2)),
    "last_column": (31, 12, 9, [[6, 0], [0, 3], [2, 2]], (26, 5, 4), (5, 3, 2)),
    "one_plane_over": (64, 8, 25, [[0, 0], [0, 0], [5, 5]], (30, 2, 12), (3, 2, 3)),
}


@pytest.mark.parametrize("precision,tol", [("f64", 1e-8), ("f32", 1e-3)])
@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("every", [STEPS, 37])
def test_gradient_matches_the_oracle(lib, oracle_lib, grid, precision, tol, every):
    inst, des, obj = case(*GRIDS[grid], seed=5)
    o = OracleFields(inst)
    o.set_design(des)
    F0, g0 = o.adjoint(obj, STEPS)
    f = Fields(inst, precision)
    f.set_design(des)
    F, g = f.adjoint_gradient(obj, STEPS, checkpoint_every=every)
    assert F[0] == pytest.approx(F0, rel=1e-10 if precision == "f64" else 1e-4)
    assert np.max(np.abs(g0)) > 0
    assert np.max(np.abs(g[0] - g0)) <= tol * np.max(np.abs(g0))
    assert f.steps_done == STEPS
    f.synchronize()


def test_unequal_designs_in_one_sim(lib):
    cases = [case(*GRIDS[k], seed=s) for s, k in enumerate(("odd", "last_column", "odd"))]
    f = Fields([c[0] for c in cases], "f32")
    for q, c in enumerate(cases):
        f.set_design(c[1], q)
    F, g = f.adjoint_gradient([c[2] for c in cases], STEPS, checkpoint_every=40)
    for q, (inst, des, obj) in enumerate(cases):
        s = Fields(inst, "f32")
        s.set_design(des)
        F1, g1 = s.adjoint_gradient(obj, STEPS, checkpoint_every=STEPS)
        assert F1[0] == F[q]
        np.testing.assert_array_equal(g1[0], g[q])


def test_memory_refused_is_what_would_not_fit(lib):
    """With 30 arrays' worth of memory free, the objective (no copies of the state) and a gradient of one segment
    (21 arrays) run; five checkpoints of 18 arrays each are refused, and the state is then as it was."""
    import torch
    inst, des, obj = adjoint_case(n=128, res=40.0, design_um=(0.2, 0.2, 0.1))
    inst.material.regions[0].susceptibilities = []
    src = inst.sources[0]
    src.start_time, src.end_time = -9.0, 11.0
    src.lo, src.hi = src.lo[:2] + (1.5,), src.hi[:2] + (1.5,)  # four cells below the patch
    f = Fields(inst, "f64")
    f.set_design(des)
    f.step(4)
    want = f.get_array(0)
    array = 128 ** 3 * 8
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - 30 * array, dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(_abi.SJError) as e:
            f.adjoint_gradient([obj], 20, checkpoint_every=4)
        assert e.value.code == _abi.SJ_E_NOMEM
        assert f.steps_done == 4
        np.testing.assert_array_equal(f.get_array(0), want)
        F = f.objective([obj], 20)
        Fg, g = f.adjoint_gradient([obj], 20, checkpoint_every=0)
        assert Fg[0] == F[0] and np.max(np.abs(g[0])) > 0 and f.steps_done == 20
    finally:
        del hog
        torch.cuda.empty_cache()
    f.close()


@pytest.mark.parametrize("cells,comps", [(21, (0, 1, 2)), (22, (0, 1, 2)), (627, (2,)), (33 * 19 * 17, (0, 2))])
def test_objectives_of_many_cells(lib, oracle_lib, cells, comps):
    """The objective's source over one block, a block and a remainder, more blocks than z segments, and every cell."""
    inst, des, _ = case(*GRIDS["odd"], seed=7)
    q = np.arange(cells)
    obj = Objective(np.stack([q % 33, q // 33 % 19, (8 + q // 627) % 17], axis=1), frequency=1 / 0.7, comps=comps)
    o = OracleFields(inst)
    o.set_design(des)
    F0, g0 = o.adjoint(obj, STEPS)
    f = Fields(inst, "f64")
    f.set_design(des)
    F, g = f.adjoint_gradient(obj, STEPS, checkpoint_every=STEPS)
    assert F[0] == pytest.approx(F0, rel=1e-10)
    assert np.max(np.abs(g0)) > 0
    assert np.max(np.abs(g[0] - g0)) <= 1e-8 * np.max(np.abs(g0))
