"""The cooperative kernels on mechanisms of up to a warp's species, which one warp solves: FP64 bit for bit against
the oracle, mixed within 1e-6 of it, at the edges of the eight columns that are loaded ahead."""
import numpy as np
import pytest

import simstack_gb300 as sg

from test_gpu_coop import assert_state, synthetic_pair

pytestmark = pytest.mark.gpu

CTL = dict(rtol=1e-4, atol=1e-12, max_steps=200000)


@pytest.mark.parametrize("n,R", [(2, 3), (3, 6), (7, 14), (8, 24), (9, 27), (16, 48), (17, 60), (24, 80), (31, 100), (32, 110)])
def test_up_to_a_warp(module, oracle_lib, n, R):
    pm, om = synthetic_pair(oracle_lib, 5, n, R)
    module.coop_set_mech(pm, sg.method("rodas3"), sg.control(**CTL))
    z0 = sg.synthetic_cells(pm, 5, seed=n)
    ref = z0.copy()
    om.advance("rodas3", oracle_lib.control(**CTL), ref.as_dict(), ref.padded, 0, 5, 1e-3, 0, 5)
    z, zm = z0.copy(), z0.copy()
    module.coop_integrate(z, 1e-3, precision=0, lane_count=5)
    assert_state(z, ref, 5)
    module.coop_integrate(zm, 1e-3, precision=2, lane_count=5)
    a, b = zm["y"][:, :5], ref["y"][:, :5]
    assert zm["failed"][:5].max() == 0.0
    assert (np.abs(a - b) / np.maximum(np.abs(b), 1e-12)).max() < 1e-6
    module.reset_arena()
