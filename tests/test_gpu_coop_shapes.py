"""The cooperative kernels where their panels and solves have remainders: species counts around the
panel widths (4, 8), the warp (32) and the smallest panelled mechanism, at one thread per row and
with fewer threads than rows (which keeps the pivot-by-pivot elimination). FP64 bit for bit
against the oracle; mixed at both thread counts the same bits as each other where the order of
operations is the same, and within 1e-6 of FP64."""
import numpy as np
import pytest

import simstack_gb300 as sg

from test_gpu_coop import assert_state, synthetic_pair

pytestmark = pytest.mark.gpu

CTL = dict(rtol=1e-4, atol=1e-12, max_steps=200000)


@pytest.fixture
def shapes():
    yield sg.lib().gpu_kin_coop_set_shape
    sg.lib().gpu_kin_coop_set_shape(0, 256, 2)   # the defaults
    sg.lib().gpu_kin_coop_set_shape(2, 512, 1)


@pytest.mark.parametrize("n,R", [(33, 120), (39, 160), (40, 160), (41, 200), (63, 300), (64, 320), (65, 320), (97, 500), (130, 700),
                                 (201, 1000)])
def test_remainders(module, oracle_lib, shapes, n, R):
    pm, om = synthetic_pair(oracle_lib, 11, n, R)
    module.coop_set_mech(pm, sg.method("rodas3"), sg.control(**CTL))
    z0 = sg.synthetic_cells(pm, 5, seed=n)
    ref = z0.copy()
    om.advance("rodas3", oracle_lib.control(**CTL), ref.as_dict(), ref.padded, 0, 5, 1e-4, 0, 5)
    mixed = []
    for block in (64, 256 if n > 128 else 128):
        assert shapes(0, block, 1) == 0 and shapes(2, block, 1) == 0
        z, zm = z0.copy(), z0.copy()
        module.coop_integrate(z, 1e-4, precision=0, lane_count=5)
        assert_state(z, ref, 5)
        module.coop_integrate(zm, 1e-4, precision=2, lane_count=5)
        a, b = zm["y"][:, :5], ref["y"][:, :5]
        assert zm["failed"][:5].max() == 0.0
        assert (np.abs(a - b) / np.maximum(np.abs(b), 1e-12)).max() < 1e-6
        mixed.append(zm)
    assert np.array_equal(mixed[0]["y"], mixed[1]["y"]) and np.array_equal(mixed[0]["h"], mixed[1]["h"])
    module.reset_arena()
