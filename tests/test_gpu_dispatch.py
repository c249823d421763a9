"""Which launches a call takes must not change what it accepts or returns."""
import numpy as np
import pytest

from sim_juncs_gb300 import _abi
from sim_juncs_gb300.configs import junction_instance
from sim_juncs_gb300.fields import Fields
from sim_juncs_gb300.geometry import Box
from sim_juncs_gb300.spec import PML, Grid, Probe, Region, Scene

pytestmark = pytest.mark.gpu


def equal_sims(a, b):
    assert a.steps_done == b.steps_done
    for q in range(a.n_instances):
        for c in range(6):
            np.testing.assert_array_equal(a.get_array(c, q), b.get_array(c, q), err_msg=f"instance {q} component {c}")
        np.testing.assert_array_equal(a.monitors(q), b.monitors(q))
        np.testing.assert_array_equal(a.dft(q), b.dft(q))


def lit(f, inst=0):
    return max(float(np.max(np.abs(f.get_array(c, inst)))) for c in range(6)) > 0


def column(nz):
    """A long thin cell: few tiles, many planes; a box and a sheet near one end."""
    inst = junction_instance(n=32, res=20.0)
    dx = inst.grid.dx
    inst.grid = Grid(32, 8, nz, dx, inst.grid.dt)
    inst.pml = PML([[0.0, 0.0], [0.0, 0.0], [0.2, 0.2]])
    inst.material = Scene([Region(Box((0.4, 0.0, 1.0), (1.2, 0.4, 1.3)), eps=2.0)], ambient_eps=1.0)
    src = inst.sources[0]
    src.start_time, src.end_time = -9.0, 11.0
    src.lo, src.hi = (0.0, 0.0, 0.8), (32 * dx, 8 * dx, 0.8)
    inst.probes = [Probe(0, (0.8, 0.2, 0.9), dft=True)]
    return inst


@pytest.mark.parametrize("nz", [8192, 8193, 16384])
def test_long_thin_grids_take_single_steps(lib, nz):
    # more than 8192 planes do not fit the tile codes in segments of 8
    a, b = Fields(column(nz), "f32"), Fields(column(nz), "f32")
    b.set_tiling(8, 0, 16)
    assert a.launches_per_step() > 0
    for f in (a, b):
        f.step(1)
        f.step(20)
        f.step_graph(1, chunk=1)
    equal_sims(a, b)
    assert lit(a)
    a.close()
    b.close()


def test_no_steps_ask_for_nothing(lib):
    # more planes than any tile code names: runs need no tiles, single steps are refused, no steps are nothing
    f = Fields(column(16385), "f64")
    f.set_tiling(8, 0, 16)
    f.step(0)
    with pytest.raises(_abi.SJError) as e:
        f.step(1)
    assert e.value.code == _abi.SJ_E_INVALID and f.steps_done == 0
    f.close()
    f = Fields(column(16385), "f64")   # (in FP32 it has more cells than resident runs take)
    f.step(0)
    f.step(3)
    assert f.steps_done == 3 and lit(f)
    f.close()


@pytest.mark.parametrize("warm", [(1,) * 40, (30, 10)], ids=["single", "runs"])
@pytest.mark.parametrize("captured", [(1, 1), (6,)], ids=["single", "run"])
def test_warmed_up_sims_can_be_captured(lib, warm, captured):
    # the warm-up's kind of call (single steps or runs) need not be the captured one
    import torch
    s = torch.cuda.Stream()
    inst = junction_instance(n=40, res=12.5, dft=False, probe_components=())
    a, b = Fields(inst, "f32", stream=s), Fields(inst, "f32")
    for n in warm:
        a.step(n)
    a.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for n in captured:
            a.step(n)
    with torch.cuda.stream(s):
        for _ in range(3):
            g.replay()
    s.synchronize()
    b.step(sum(warm) + 3 * sum(captured))
    for c in range(6):
        np.testing.assert_array_equal(a.get_array(c), b.get_array(c))
    assert lit(a)
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_single_step_graphs_between_runs(lib, precision):
    # single steps replay graphs of the tile launches, one per parity; runs step in place
    insts = [junction_instance(n=n, res=r, phase=p) for n, r, p in ((40, 12.5, 0.3), (64, 20.0, 1.0), (40, 12.5, 2.0))]
    for i in insts:
        i.sources[0].start_time, i.sources[0].end_time = -9.0, 11.0
    a, b = Fields(insts, precision), Fields(insts, precision)
    b.set_tiling(8, 0, 8)
    for _ in range(5):
        a.step_graph(1, chunk=1)
    a.step(7)
    for _ in range(4):
        a.step_graph(1, chunk=1)
    a.step_graph(20, chunk=1)
    a.step(1)
    a.step_graph(1, chunk=1)
    b.step(38)
    equal_sims(a, b)
    assert lit(a)
    a.close()
    b.close()


def test_launch_counts_follow_the_dispatch(lib):
    inst = junction_instance(n=64, res=20.0)
    f = Fields(inst, "f32")
    one = f.launches_per_step()
    assert f.run_launches(1) == one and f.run_launches(0) == 0
    assert f.run_launches(2) == f.run_launches(256) == 1 and f.run_launches(257) == 2
    f.set_tiling(*f.tiling())                       # asks for the tile launches
    assert f.run_launches(256) == 256 * one
    f.close()
    big = Fields(junction_instance(n=192, res=60.0), "f32")
    assert big.run_launches(10) == 10 * big.launches_per_step()
    big.close()
    inst.probes = [Probe(0, (1.6, 1.6, 1.6), dft=True)] * 60000
    inst.freqs = list(np.linspace(1.0, 2.0, 50))    # the probes outweigh what a resident run gains
    f = Fields(inst, "f32")
    assert f.run_launches(10) == 10 * f.launches_per_step()
    f.close()


@pytest.mark.parametrize("precision,mode", [("f32", "grouped"), ("f32", "queue"), ("f64", "grouped")])
def test_autotune_keeps_resident_runs(lib, precision, mode):
    # poles, psi and DFT sums are stepped in place: timing a run must leave them as they were
    insts = [junction_instance(n=64, res=20.0, phase=p) for p in (0.4, 1.9)]
    for i in insts:
        i.sources[0].start_time, i.sources[0].end_time = -9.0, 11.0
    a, b = Fields(insts, precision), Fields(insts, precision)
    a.step(31)
    b.step(31)
    a.set_fused_launch(mode)
    ms = a.autotune(2)[3]
    assert ms > 0 and a.fused_launch() == "grouped" and a.run_launches(256) == 1
    a.synchronize()
    for n in (1, 40):
        a.step(n)
        b.step(n)
    equal_sims(a, b)
    assert lit(a)
    a.close()
    b.close()


def test_threads_step_their_own_sims(lib):
    # tables and buffers that grow while other threads copy and step: each sim's kernels see its own
    from concurrent.futures import ThreadPoolExecutor
    jobs = [(junction_instance(n=n, res=r, phase=0.3 * q), p, tiles)
            for q, (n, r, p, tiles) in enumerate([(36, 11.25, "f32", False), (64, 20.0, "f64", False), (48, 15.0, "f32", True),
                                                  (64, 20.0, "f64", False), (36, 11.25, "f64", True), (64, 20.0, "f32", False)])]

    def run(job):
        inst, precision, tiles = job
        f = Fields(inst, precision)
        if tiles:
            f.set_tiling(8, 0, 8)
        for n in (1, 2, 5, 12, 30, 70, 160, 300):
            f.step(n)
        out = [f.get_array(c) for c in range(6)] + [f.monitors(), f.dft()]
        f.close()
        return out

    want = [run(j) for j in jobs]
    assert all(max(np.max(np.abs(a)) for a in w[:6]) > 0 for w in want)
    for _ in range(5):
        with ThreadPoolExecutor(len(jobs)) as ex:
            for w, g in zip(want, ex.map(run, jobs)):
                for x, y in zip(w, g):
                    np.testing.assert_array_equal(x, y)
