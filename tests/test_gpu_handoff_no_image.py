"""Straggler hand-off of a mechanism whose schedule image the group kernels do not have (a net change of 33
fits no term word): the cooperative kernel finishes the cells, with the oracle's bits."""
import ctypes as C

import numpy as np
import pytest

import simstack_gb300 as sg

pytestmark = pytest.mark.gpu

CTL = dict(rtol=1e-4, atol=1e-12, max_steps=2000)


def model(O):
    pm, om = sg.Model.new(), O.Mechanism()
    rates = []
    for s in range(6):
        pm.add_species(f"S{s}", True)
        om.add_species(f"S{s}", True)
    for eq, k in (("S0 + S1 -> " + " + ".join(["S2"] * 33), 1e3), ("S2 -> S3", 1e4), ("S3 + S4 -> S5", 1e7), ("S5 -> S0 + S1", 10.0), ("S3 -> S4", 1.0)):
        pm.add_reaction(eq, "arr", (k, 0.0, 0.0))
        om.add_reaction(eq, "arr", (k, 0.0, 0.0))
        rates.append(k)
    pm.finalize()
    om.finalize()
    pm.k_const = np.array(rates)
    return pm, om


@pytest.mark.parametrize("block", [32, 128])
@pytest.mark.parametrize("kind", [0, 2])
def test_parked_and_finished(module, oracle_lib, kind, block):
    pm, om = model(oracle_lib)
    km = pm.kinmech()
    assert sg.lib().kin_mech_group_image(C.byref(km), 32, 0, None, 0) == 0
    z = sg.synthetic_cells(pm, 300, seed=4)
    ref = z.copy()
    module.set_mech(km, sg.method("rodas3"), sg.control(**CTL))
    module.set_tuning(kind=kind)
    module.set_straggler_budget(30)
    sg.check(sg.lib().gpu_kin_set_straggler_block(block), "gpu_kin_set_straggler_block")
    try:
        module.integrate(z, 0.1, precision=0)
        parked = module.parked_cells()
    finally:
        module.set_straggler_budget(sg.DEFAULT_STRAGGLER_BUDGET)
        sg.check(sg.lib().gpu_kin_set_straggler_block(128), "gpu_kin_set_straggler_block")
        sg.check(sg.lib().gpu_init(0, 2 << 30, module.info), "gpu_init")   # no tuning set
    om.advance("rodas3", oracle_lib.control(**CTL), ref.as_dict(), ref.padded, 0, ref.padded, 0.1, 0, 0)
    assert parked > 0
    for name in ("y", "h", "steps", "rejects", "pulses", "failed"):
        assert z[name].tobytes() == ref[name].tobytes(), f"{name}: {np.count_nonzero(z[name] != ref[name])} differ"
