"""The lane-group kernels (8, 16 or 32 lanes per cell), which the module chooses by batch size until a
tuning is set: the same bits as the oracle (FP64, f32) and as the oracle's model of the mixed path, at
the sizes where the rule changes shape, on mechanisms of each size class, and where a warp hands its
last cell to all its lanes."""
import numpy as np
import pytest

import simstack_gb300 as sg

from test_gpu_parity import DBD_CTL, assert_bits, oracle_run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def untuned(module):
    """The module as gpu_init leaves it (no tuning set): the rule by size is in force."""
    sg.check(sg.lib().gpu_init(0, 2 << 30, module.info), "gpu_init")
    yield module
    sg.check(sg.lib().gpu_init(0, 2 << 30, module.info), "gpu_init")


def oracle_advance(O, z, duration, precision, method="rodas3", ctl=None, mech=None):
    if precision != 2:
        oracle_run(O, z, duration, precision, method, O.control(**ctl) if ctl else None, mech)
        return
    m = mech if mech is not None else O.Mechanism.air()
    O.advance_mixed(m, method, O.control(**(ctl or {})), z.as_dict(), z.padded, 0, z.padded, duration, sweeps=1, variant=2)


# cells: one, a few, 32 lanes per cell (<= 8 or 10 per SM), 16 (<= 16 or 26), 8 (<= 96 or 48), and one lane
@pytest.mark.parametrize("precision", [0, 2])
# (FP64: CTAs of 1, 1, 5, 6, 5, 8 and 4 warps)
@pytest.mark.parametrize("cells", [1, 3, 613, 1601, 2801, 4801, 5003])
def test_shipped_mechanism_by_size(untuned, oracle_lib, cells, precision):
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control())
    z = sg.air_cells(cells, seed=cells)
    ref = z.copy()
    untuned.integrate(z, 0.5, precision=precision)
    oracle_advance(oracle_lib, ref, 0.5, precision)
    assert_bits(z, ref)
    untuned.reset_arena()


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("cells", [5, 700, 1700])
def test_pulsed_zones(untuned, oracle_lib, cells, precision):
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control(**DBD_CTL))
    i = np.arange(cells)
    z = sg.dbd_zones(cells, 300.0 + 10.0 * (i % 5), 0.005 * (i % 7), 0.05 + 0.1 * (i % 3), 5000.0 + 2500.0 * (i % 4))
    sg.dbd_prepare_source(z, True, 0.0, 5e-4)
    ref = z.copy()
    untuned.integrate(z, 5e-4, precision=precision)
    oracle_advance(oracle_lib, ref, 5e-4, precision, ctl=DBD_CTL)
    assert_bits(z, ref)
    assert z["pulses"].min() > 0
    untuned.reset_arena()


SYN_CTL = dict(rtol=1e-4, atol=1e-12, max_steps=200000)


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("n,R,seed,cells,method", [(3, 6, 2, 40, "ros2"), (12, 40, 1, 1300, "rodas3"), (20, 60, 1, 100, "ros3"),
                                                   (24, 80, 5, 2500, "rodas3"), (32, 64, 1, 300, "rodas3")])
def test_table_mechanisms(untuned, oracle_lib, n, R, seed, cells, method, precision):
    pm = sg.Model.synthetic(seed=seed, species=n, reactions=R, bimolecular=0.7, products=1)
    om = oracle_lib.Mechanism()
    for s in range(n):
        om.add_species(f"S{s}", True)
    for r in range(pm.R):
        om.add_reaction(sg.model_equation(pm, r), "arr", (float(pm.k_const[r]), 0.0, 0.0))
    om.finalize()
    untuned.set_mech(pm.kinmech(), sg.method(method), sg.control(**SYN_CTL))
    z = sg.synthetic_cells(pm, cells, seed=3)
    ref = z.copy()
    untuned.integrate(z, 0.1, precision=precision)
    oracle_advance(oracle_lib, ref, 0.1, precision, method, SYN_CTL, om)
    assert_bits(z, ref)
    untuned.reset_arena()


@pytest.mark.parametrize("precision", [0, 2])
def test_stiff_cells_reach_a_whole_warp(untuned, oracle_lib, precision):
    """Uneven stiffness with a low budget: warps stop claiming for a long cell and hand it to all lanes."""
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control())
    untuned.set_straggler_budget(60)
    z = sg.air_cells(3001, seed=3)
    sg.air_source(z, seed=3, P0=1e-2, decades=3.0)
    ref = z.copy()
    untuned.integrate(z, 5.0, precision=precision)
    untuned.set_straggler_budget(sg.DEFAULT_STRAGGLER_BUDGET)
    oracle_advance(oracle_lib, ref, 5.0, precision)
    assert_bits(z, ref)
    untuned.reset_arena()


def test_failed_and_subset_lanes(untuned, oracle_lib):
    """A step cap that some cells reach, and a lane_count below the padding: the rest is untouched."""
    ctl = dict(max_steps=40)
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control(**ctl))
    z = sg.air_cells(256, seed=2)
    ref = z.copy()
    base = untuned.upload(z)
    untuned.advance(z.launch(base, 0, 1.0, lane_count=201))
    untuned.download(z, base)
    oracle_lib.Mechanism.air().advance("rodas3", oracle_lib.control(**ctl), ref.as_dict(), ref.padded, 0, 201, 1.0, 0, 0)
    assert_bits(z, ref)
    assert z["failed"].sum() > 0
    untuned.reset_arena()


@pytest.mark.parametrize("precision,cells", [(0, 12001), (2, 6501), (2, 19999), (1, 5001)])
def test_large_batches_by_rule(untuned, cells, precision):
    """Past the group kernels' range: the lane shapes the rule picks, whose last cells are parked and resumed
    (FP64, mixed), against the warp-synchronous queue, which parks none with the hand-off off."""
    ctl = DBD_CTL if precision == 1 else {}
    z = sg.air_cells(cells, seed=7)
    ref = z.copy()
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control(**ctl))
    dur = 1e-4 if precision == 1 else 0.3
    untuned.integrate(z, dur, precision=precision)
    if precision != 1:
        assert untuned.parked_cells() > 0
    untuned.reset_arena()
    untuned.set_straggler_budget(0)
    untuned.set_tuning(kind=1)
    untuned.integrate(ref, dur, precision=precision)
    untuned.set_straggler_budget(sg.DEFAULT_STRAGGLER_BUDGET)
    sg.check(sg.lib().gpu_init(0, 2 << 30, untuned.info), "gpu_init")   # untuned again
    assert_bits(z, ref)


@pytest.mark.parametrize("precision,kind,cells", [(0, 2, 700), (2, 4, 700), (0, 2, 16001)])
def test_autotune_against_the_rule(untuned, oracle_lib, precision, kind, cells):
    """An autotuned small batch keeps the rule's group kernel (no lane shape is near it), a large one takes the
    measured lane shape; the same bits."""
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control())
    z = sg.air_cells(cells, seed=9)
    ref = z.copy()
    base = untuned.upload(z)
    t = untuned.autotune(z.launch(base, precision, 0.2), kind=kind)
    ms = untuned.advance(z.launch(base, precision, 0.2))
    if cells == 700:
        assert ms < t.ms
    untuned.download(z, base)
    sg.check(sg.lib().gpu_init(0, 2 << 30, untuned.info), "gpu_init")   # untuned again
    oracle_advance(oracle_lib, ref, 0.2, precision)
    assert_bits(z, ref)
