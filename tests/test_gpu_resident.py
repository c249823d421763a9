"""Small grids step through one cooperative launch per run of steps; the tile
kernels (which an explicit set_tiling asks for, and which single steps use)
must give the same bits: same arithmetic per cell, other work split."""
import numpy as np
import pytest

from sim_juncs_gb300 import _abi
from sim_juncs_gb300.configs import inverse_design_case, junction_instance
from sim_juncs_gb300.fields import Fields
from sim_juncs_gb300.spec import PML, Grid, Probe

pytestmark = pytest.mark.gpu


def odd_box():
    """Odd, unequal sides; slabs on some faces only; an Hy sheet; H and E probes sampled every 3 steps."""
    inst = junction_instance(n=45, res=14.0, probe_components=("Ex", "Hy", "Hz"), component=_abi.HY, save_span=3)
    inst.grid = Grid(37, 45, 29, inst.grid.dx, inst.grid.dt)
    inst.pml = PML([[0.3, 0.0], [0.0, 0.4], [0.25, 0.25]])
    return [inst]


def whole_slab():
    """Every column in an x slab, one plane of cells in z, no probes."""
    inst = junction_instance(n=20, res=14.0)
    inst.grid = Grid(8, 20, 1, inst.grid.dx, inst.grid.dt)
    inst.pml = PML([[4 / 14.0, 4 / 14.0], [0.0, 0.0], [0.0, 0.0]])
    inst.probes, inst.freqs = [], []
    return [inst]


def many_probes():
    """More probes than the probe blocks hold one each (several chunks per block), on two of three grids."""
    a, b = junction_instance(n=32, res=10.0), junction_instance(n=33, res=10.5, probe_components=("Ez",), dft=False)
    a.probes = [Probe(c, (0.3 + 0.0003 * q, 1.6, 1.6), dft=c != _abi.EZ) for c in (0, 2, 4) for q in range(3800)]
    return [a, junction_instance(n=24, res=7.5, probe_components=(), dft=False), b]


def batch():
    return [junction_instance(n=n, res=r, phase=ph, amplitude=am) for n, r, ph, am in
            ((64, 20.0, 0.3, 2.0), (40, 12.5, 1.7, 0.5), (64, 20.0, 4.0, 1.0))]


def mostly_plain():
    """Rows of whole tiles and mostly plain tiles: the tile launches keep their classes (elsewhere here they merge)."""
    inst = junction_instance(n=96, res=30.0)
    inst.grid = Grid(128, 24, 128, inst.grid.dx, inst.grid.dt)
    inst.pml = PML([[0.1, 0.0], [0.0, 0.0], [0.1, 0.1]])
    src = inst.sources[0]
    src.start_time, src.end_time = -9.0, 11.0
    src.lo, src.hi = (0.0, 0.0, 1.7), (4.3, 0.8, 1.7)
    inst.probes = [Probe(c, (2.0, 0.4, z), dft=True) for c in (0, 4) for z in (0.05, 2.0)]
    return [inst]


CASES = {"mostly_plain": mostly_plain, "odd_box": odd_box, "whole_slab": whole_slab, "many_probes": many_probes, "batch": batch,
         "quartz": lambda: [inverse_design_case(0, n=72)[0]], "junction65": lambda: [junction_instance(n=65, res=20.0)]}


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("case", CASES)
def test_resident_runs_equal_tile_launches(lib, case, precision):
    insts = CASES[case]()
    a, b = Fields(insts, precision), Fields(insts, precision)
    b.set_tiling(8, 0, 8)
    for n in (3, 1, 290, 2):  # odd parities, a single (tile) step between runs, a run longer than one launch
        a.step(n)
    a.step_graph(7, chunk=2)
    b.step(303)
    assert a.steps_done == b.steps_done == 303
    a.synchronize()
    for q in range(len(insts)):
        for c in range(6):
            np.testing.assert_array_equal(a.get_array(c, q), b.get_array(c, q), err_msg=f"instance {q} component {c}")
        np.testing.assert_array_equal(a.monitors(q), b.monitors(q))
        np.testing.assert_array_equal(a.dft(q), b.dft(q))
    assert case == "whole_slab" or max(float(np.max(np.abs(a.get_array(c)))) for c in range(6)) > 0
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_design_and_objective_through_both_paths(lib, precision):
    """Design cells, their recorded brackets (one and several segments) and the objective's sums, two designs of
    which one has more objective cells than a block has threads."""
    cases = [inverse_design_case(q, n=72, design_um=(0.4, 0.3, 0.1), patch=p) for q, p in ((0, 5), (1, 19))]
    for inst, _, _ in cases:
        inst.sources[0].start_time, inst.sources[0].end_time = -9.0, 11.0
    out = []
    for tiles in (False, True):
        f = Fields([c[0] for c in cases], precision)
        if tiles:
            f.set_tiling(8, 0, 16)
        for q, c in enumerate(cases):
            f.set_design(c[1], q)
        f.step(60)
        grads = [f.adjoint_gradient([c[2] for c in cases], 61, checkpoint_every=k) for k in (20, 61)]
        out.append((f.objective([c[2] for c in cases], 40), grads, [f.get_array(c, q) for q in (0, 1) for c in range(6)]))
        f.close()
    assert out[0][0].min() > 0
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for (Fa, ga), (Fb, gb) in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(Fa, Fb)
        for x, y in zip(ga, gb):
            assert np.max(np.abs(x)) > 0
            np.testing.assert_array_equal(x, y)
    for x, y in zip(out[0][2], out[1][2]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("counts,freqs", [((1000,), 50), ((33,), 20), ((700, 31, 0, 400), 30), ((9000,), 40)],
                         ids=["small chunks", "one over a warp", "several grids", "more than pays"])
def test_probes_dealt_out_over_blocks(lib, precision, counts, freqs):
    """Probe blocks with fewer probes than threads, chunks that end inside an instance, instances without probes, and
    so many that the run goes to the tile launches: every sum as the tile launches form it."""
    rng = np.random.default_rng(3)
    insts = []
    for n in counts:
        inst = junction_instance(n=36, res=11.25, probe_components=(), save_span=2)
        inst.sources[0].start_time, inst.sources[0].end_time = -9.0, 11.0
        at = rng.uniform(0.3, 2.9, size=(n, 3))
        inst.probes = [Probe((0, 4, 2, 3)[q % 4], tuple(at[q]), monitor=q % 5 == 0, dft=q % 7 != 0) for q in range(n)]
        inst.freqs = list(np.linspace(0.8, 2.0, freqs))
        insts.append(inst)
    a, b = Fields(insts, precision), Fields(insts, precision)
    b.set_tiling(8, 0, 8)
    for n in (21, 1, 20):
        a.step(n)
    b.step(42)
    for q in range(len(insts)):
        np.testing.assert_array_equal(a.monitors(q), b.monitors(q))
        np.testing.assert_array_equal(a.dft(q), b.dft(q))
        assert not len(insts[q].probes) or np.max(np.abs(a.dft(q))) > 0
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_every_column_in_a_slab(lib, precision):
    """Grids of one plane and of a few whose every column lies in an x slab, the sheet inside them."""
    insts = []
    for nz in (1, 5):
        inst = whole_slab()[0]
        inst.grid = Grid(8, 20, nz, inst.grid.dx, inst.grid.dt)
        src = inst.sources[0]
        src.start_time, src.end_time = -9.0, 11.0
        src.lo, src.hi = (0.0, 0.0, 0.0), (8 / 14.0, 20 / 14.0, 0.0)
        insts.append(inst)
    a, b = Fields(insts, precision), Fields(insts, precision)
    b.set_tiling(8, 0, 8)
    a.step(41)
    b.step(41)
    for q in (0, 1):
        for c in range(6):
            np.testing.assert_array_equal(a.get_array(c, q), b.get_array(c, q), err_msg=f"instance {q} component {c}")
        assert all(np.max(np.abs(a.get_array(c, q))) > 0 for c in ((0, 5) if q == 0 else (0, 4, 5)))
    a.close()
    b.close()
