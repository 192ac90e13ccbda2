"""Mixed cooperative kernels where FP32 overflows: a lane past the last species takes no part in a solve."""
import numpy as np
import pytest

import simstack_gb300 as sg

pytestmark = pytest.mark.gpu


@pytest.fixture
def shapes():
    yield sg.lib().gpu_kin_coop_set_shape
    sg.lib().gpu_kin_coop_set_shape(2, 512, 1)   # the default


def chains(n, split, closing=None):
    """S0 -> S1 -> .. and, apart from it, S{split} -> .. -> S{n-1}; closing: and S{n-1} -> S0 at this rate."""
    m = sg.Model.new()
    for s in range(n):
        m.add_species(f"S{s}", True)
    k = []
    for s in range(n - 1):
        if s + 1 != split:
            m.add_reaction(f"S{s} -> S{s + 1}")
            k.append(0.5 + s % 5)
    if closing:
        m.add_reaction(f"S{n - 1} -> S0")
        k.append(closing)
    m.finalize()
    z = sg.ZoneBlock(n, m.R, 3)
    z["k"][:] = np.array(k)[:, None]
    z["y"][:] = 1e-3 * (1.0 + np.arange(n) % 7)[:, None]
    return m, z


def panels_and_pattern(module, shapes, m, z0, ctl, duration):
    """The block after an advance with a thread per species, and with fewer (which tests every element's
    pattern)."""
    out = []
    module.coop_set_mech(m, sg.method("rodas3"), ctl)
    for block in (128, 64):
        assert shapes(2, block, 1) == 0
        z = z0.copy()
        module.coop_integrate(z, duration, precision=2, lane_count=3)
        module.reset_arena()
        out.append(z)
    return out


@pytest.mark.parametrize("n", [65, 66, 95])
def test_lanes_past_the_last_species(module, shapes, n):
    """U(0, n-1) x[n-1] of the forward pass is past FP32's range; no row of the mechanism forms it."""
    m, z = chains(n, n, closing=1e20)
    z["y"][n - 1] = 0.1
    a, b = panels_and_pattern(module, shapes, m, z, sg.control(rtol=1e-4, atol=1e-12, max_steps=40), 1e-9)
    assert np.isfinite(b["y"]).all() and b["failed"].max() == 0.0
    for name in ("y", "h", "steps", "rejects", "failed"):
        assert np.array_equal(a[name][..., :3], b[name][..., :3]), name
