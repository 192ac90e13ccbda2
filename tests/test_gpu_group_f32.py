"""The f32 group kernels (table mechanisms) bit for bit against the oracle, for every size of kernel and number
of lanes per cell; and the group kernels behind the pipelined and asynchronous advances, where chunks run on
two streams. No tuning is set, so the rule by size chooses."""
import ctypes as C

import numpy as np
import pytest

import simstack_gb300 as sg

from test_gpu_group import oracle_advance, untuned  # noqa: F401
from test_gpu_parity import assert_bits

pytestmark = pytest.mark.gpu

CTL = dict(rtol=1e-3, atol=1e-12, max_steps=300)


def mechanism(O, n, R, seed):
    pm = sg.Model.synthetic(seed=seed, species=n, reactions=R, bimolecular=0.7, products=1)
    om = O.Mechanism()
    for s in range(n):
        om.add_species(f"S{s}", True)
    for r in range(pm.R):
        om.add_reaction(sg.model_equation(pm, r), "arr", (float(pm.k_const[r]), 0.0, 0.0))
    om.finalize()
    return pm, om


# kernels of at most 12, exactly 17 (Rodas3), at most 20 and 32 species; 32 lanes per cell up to 11 cells per SM, 16 up to
# 16, then 8
@pytest.mark.parametrize("cells", [1, 301, 2001, 2603])
@pytest.mark.parametrize("n,R,seed,method", [(3, 6, 2, "rodas3"), (12, 40, 1, "ros2"), (17, 50, 4, "rodas3"), (17, 50, 4, "ros3"), (20, 60, 1, "rodas3"),
                                             (24, 80, 5, "ros3"), (32, 64, 1, "rodas3")])
def test_f32_table_mechanisms(untuned, oracle_lib, n, R, seed, method, cells):  # noqa: F811
    pm, om = mechanism(oracle_lib, n, R, seed)
    untuned.set_mech(pm.kinmech(), sg.method(method), sg.control(**CTL))
    z = sg.synthetic_cells(pm, cells, seed=3)
    ref = z.copy()
    untuned.integrate(z, 0.01, precision=1)
    oracle_advance(oracle_lib, ref, 0.01, 1, method, CTL, om)
    assert_bits(z, ref)
    assert z["steps"].min() > 0
    untuned.reset_arena()


@pytest.mark.parametrize("chunks", [2, 5])
@pytest.mark.parametrize("precision,n", [(0, 17), (1, 8), (2, 17), (2, 8)])
def test_pipelined_groups(untuned, oracle_lib, precision, n, chunks):  # noqa: F811
    """17 species: the shipped mechanism; 8: a table mechanism."""
    if n == 17:
        pm, om, ctl, z, dur = sg.Model.air(), None, {}, sg.air_cells(2000, seed=8), 0.2
    else:
        pm, om = mechanism(oracle_lib, 8, 24, 7)
        ctl, z, dur = CTL, sg.synthetic_cells(pm, 2000, seed=8), 0.01
    untuned.set_mech(pm.kinmech(), sg.method("rodas3"), sg.control(**ctl))
    ref = z.copy()
    untuned.integrate_pipelined(z, dur, precision=precision, chunks=chunks)
    oracle_advance(oracle_lib, ref, dur, precision, "rodas3", ctl, om)
    assert_bits(z, ref)
    untuned.reset_arena()


@pytest.mark.parametrize("precision", [0, 2])
def test_async_group(untuned, oracle_lib, precision):  # noqa: F811
    untuned.set_mech(sg.Model.air().kinmech(), sg.method("rodas3"), sg.control())
    z = sg.air_cells(1200, seed=6)
    ref = z.copy()
    base = untuned.alloc(z.nbytes)
    launch = z.launch(base, precision, 0.2)
    L = sg.lib()
    sg.check(L.gpu_kin_advance_async(C.byref(launch), z.data.ctypes.data, base, z.rows, z.mutable_rows), "gpu_kin_advance_async")
    kms, tms = C.c_float(), C.c_float()
    sg.check(L.gpu_kin_wait(C.byref(kms), C.byref(tms)), "gpu_kin_wait")
    oracle_advance(oracle_lib, ref, 0.2, precision)
    assert_bits(z, ref)
    untuned.reset_arena()
