"""Mixed cooperative kernels with values past FP32's range inside the mechanism: what is not finite stays
with the species it reaches through the mechanism's own entries (a step accepted whatever its error shows it)."""
import numpy as np
import pytest

import simstack_gb300 as sg

from test_gpu_coop_overflow import chains, panels_and_pattern, shapes  # noqa: F401

pytestmark = pytest.mark.gpu

SPLIT = 20   # S0..S19 and the rest share no reaction
CTL = dict(rtol=1e-4, atol=1e-12, max_steps=10, fixed_step=1, clamp_negative=0)   # (clamping makes a NaN a zero)


@pytest.mark.parametrize("n", [44, 64, 97])
@pytest.mark.parametrize("what", ["matrix", "right-hand side", "both"])
def test_other_species_stay_finite(module, shapes, n, what):
    m, z = chains(n, SPLIT)
    clean = z.copy()
    if what != "right-hand side":
        z["k"][3, 1] = 1e39     # an LU entry without a finite float
    if what != "matrix":
        z["src"][7, 1] = 1e40   # a right-hand side without one
    a, b = panels_and_pattern(module, shapes, m, z, sg.control(**CTL), 3e-9)
    c, _ = panels_and_pattern(module, shapes, m, clean, sg.control(**CTL), 3e-9)
    assert np.isfinite(b["y"][SPLIT:, :3]).all() and not np.isfinite(b["y"][:SPLIT, 1]).all()
    assert np.array_equal(b["y"][SPLIT:, :3], c["y"][SPLIT:, :3])
    assert np.array_equal(b["y"][:, 0::2], c["y"][:, 0::2])   # the cells beside it
    for name in ("y", "h", "steps", "rejects", "failed"):
        assert np.array_equal(a[name][..., :3], b[name][..., :3], equal_nan=True), name
