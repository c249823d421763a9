"""The fused schedule's tile kernels on grids whose runs of steps would be
resident launches: set_tiling asks for the tiles, so that their launches and
their graphs are what runs here, against the oracle and against one another."""
import numpy as np
import pytest

from oracle.oracle import OracleFields
from sim_juncs_gb300 import _abi
from sim_juncs_gb300.configs import inverse_design_case, junction_instance
from sim_juncs_gb300.fields import Fields
from sim_juncs_gb300.spec import PML, Grid, Probe

from test_gpu_parity import TOL64, compare_fields, rel

pytestmark = pytest.mark.gpu


def early(inst):
    src = inst.sources[0]
    src.start_time, src.end_time = -9.0, 11.0
    return inst


def tiles(insts, precision, zseg=8):
    f = Fields(insts, precision)
    f.set_tiling(8, 0, zseg)
    assert f.run_launches(50) == 50 * f.launches_per_step()
    return f


def equal_sims(a, b, qs=None):
    assert a.steps_done == b.steps_done
    for q in qs or range(a.n_instances):
        for c in range(6):
            np.testing.assert_array_equal(a.get_array(c, q), b.get_array(c, q), err_msg=f"instance {q} component {c}")
        np.testing.assert_array_equal(a.monitors(q), b.monitors(q))
        np.testing.assert_array_equal(a.dft(q), b.dft(q))
        assert max(float(np.max(np.abs(a.get_array(c, q)))) for c in range(6)) > 0


def groups():
    """Five launch groups: two 96^3 (merged in FP32, corrections on their own stream), 48^3 and 36^3 (ragged rows,
    one launch per class), a 64^3 with an H sheet (general tiles), and quartz under gold on 72^3."""
    out = [junction_instance(n=n, res=r, phase=p, amplitude=a, probe_components=("Ex", "Hy"))
           for n, r, p, a in ((96, 30.0, 0.3, 2.0), (48, 15.0, 1.1, 0.7), (96, 30.0, 2.9, 0.2), (36, 11.25, 0.5, 1.0),
                              (48, 15.0, 5.0, 3.0))]
    out.append(junction_instance(n=64, res=20.0, component=_abi.HY))
    out.append(inverse_design_case(0, n=72)[0])
    return [early(i) for i in out]


def mostly_plain():
    """Rows of whole tiles, mostly plain: its classes are launched one by one."""
    inst = junction_instance(n=96, res=30.0)
    inst.grid = Grid(128, 24, 128, inst.grid.dx, inst.grid.dt)
    inst.pml = PML([[0.1, 0.0], [0.0, 0.0], [0.1, 0.1]])
    inst.sources[0].lo, inst.sources[0].hi = (0.0, 0.0, 1.7), (4.3, 0.8, 1.7)
    inst.probes = [Probe(c, (2.0, 0.4, z), dft=True) for c in (0, 4) for z in (0.05, 2.0)]
    return [early(inst)]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("case,chunk", [(groups, 7), (groups, 1), (mostly_plain, 4)])
def test_graph_replays_equal_plain_launches(lib, precision, case, chunk):
    insts = case()
    a, b = tiles(insts, precision), tiles(insts, precision)
    a.step(59)
    b.step_graph(59, chunk=chunk)
    equal_sims(a, b)
    a.close()
    b.close()


@pytest.mark.parametrize("case", ["junction", "pml 0.2", "no pml", "uneven"])
def test_tiles_match_the_oracle(lib, oracle_lib, case):
    insts = {"junction": lambda: [junction_instance()], "pml 0.2": lambda: [junction_instance(n=80, res=25.0, pml_um=0.2)],
             "no pml": lambda: [junction_instance(n=80, res=25.0, pml_um=0.0)],
             "uneven": lambda: [junction_instance(n=n, res=r, phase=p, probe_components=("Ex", "Ez"))
                                for n, r, p in ((32, 10.0, 0.3), (45, 14.0, 1.7), (40, 12.5, 4.0))]}[case]()
    f = tiles([early(i) for i in insts], "f64", zseg=16)
    f.step(250)
    for q, inst in enumerate(insts):
        o = OracleFields(inst)
        o.step(250)
        compare_fields(f, o, TOL64, q)
        assert rel(f.monitors(q), o.monitors()) <= TOL64
        assert rel(f.dft(q), o.dft()) <= TOL64


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_grouped_members_equal_single_runs(lib, precision):
    insts = groups()
    f = tiles(insts, precision)
    f.step(60)
    for q, inst in enumerate(insts):
        s = tiles(inst, precision)
        s.step(60)
        for c in range(6):
            np.testing.assert_array_equal(f.get_array(c, q), s.get_array(c), err_msg=f"instance {q} component {c}")
        np.testing.assert_array_equal(f.monitors(q), s.monitors())
        np.testing.assert_array_equal(f.dft(q), s.dft())
        s.close()
    f.close()


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_columns_and_queued_launch_agree(lib, precision):
    insts = [early(junction_instance(n=n, res=r, phase=p, probe_components=("Ex", "Ez")))
             for n, r, p in ((96, 30.0, 0.3), (64, 20.0, 1.0), (96, 30.0, 2.9))]
    a, b = tiles(insts, precision), tiles(insts, precision)
    b.set_fused_columns(1)
    a.step(50)
    b.step(50)
    equal_sims(a, b)
    b.close()
    if precision == "f32":
        c = tiles(insts, precision)
        c.set_fused_launch("queue")
        c.step(20)
        c.step_graph(30, chunk=3)
        equal_sims(a, c)
        c.close()
    a.close()


def test_design_on_one_member_splits_its_group(lib):
    cases = [inverse_design_case(q, n=72, design_um=(0.4, 0.3, 0.1)) for q in (0, 1, 2)]
    insts = [early(c[0]) for c in cases]
    f = tiles(insts, "f32")
    grouped = f.launches_per_step()
    f.set_design(cases[1][1], 1)
    assert f.launches_per_step() > grouped
    f.step(60)
    for q, inst in enumerate(insts):
        s = tiles(inst, "f32")
        if q == 1:
            s.set_design(cases[1][1])
        s.step(60)
        for c in range(6):
            np.testing.assert_array_equal(f.get_array(c, q), s.get_array(c), err_msg=f"instance {q} component {c}")
        s.close()
    f.close()
