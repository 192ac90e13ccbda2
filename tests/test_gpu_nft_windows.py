"""Film windows on both sides of the rule that chooses the kernel (few substeps: through memory), against the
reference's operations: the same bits from either."""
import numpy as np
import pytest

import simstack_gb300 as sg

from test_gpu_nft_resident import ENV, REF, expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,cells,sites,offset,stride,substeps", [
    (2, 1, 1, 0, 3, 16), (3, 33, 33, 0, 1, 16), (2, 64, 21, 1, 3, 15), (2, 64, 21, 1, 3, 16), (2, 97, 1, 40, 0, 20), (3, 240, 80, 1, 3, 5),
    (1, 999, 300, 0, 3, 2), (1, 1500, 400, 1, 3, 0), (1, 1500, 400, 1, 3, 1), (33, 70, 20, 1, 3, 31), (33, 70, 20, 1, 3, 32)])
def test_windows_on_both_sides_of_the_rule(module, groups, cells, sites, offset, stride, substeps):
    rng = np.random.default_rng(cells)
    a = {"rows": rng.normal(0.0, 0.5, (groups, cells, 9, 8)).astype(np.float32), "hot": np.zeros((groups, cells, 4, 8), np.float32),
         "cold": np.zeros((groups, cells, 80), np.float32), "sites": np.zeros((groups, sites, 288), np.float32)}
    a["hot"][:, :, 0] = rng.uniform(0.05, 0.9, (groups, cells, 8))
    a["hot"][:, :, 3] = rng.uniform(0.0, 0.02, (groups, cells, 8))
    for off, hi in ((24, 1e-3), (32, 1e-5), (40, 1e-6), (48, 1e-9)):
        a["cold"][:, :, off:off + 8] = rng.uniform(0.0, hi, (groups, cells, 8))
    a["sites"][:, :, 24:88] = rng.uniform(0.0, 30.0, (groups, sites, 64))
    nt = sg.NftTransport(module, groups, cells, sites, offset, stride)
    for name, v in a.items():
        nt.upload(name, v.ravel())
    nt.run(REF, *ENV, substeps, flush_denormals=False)
    want = expected(a, cells, sites, offset, stride, substeps)
    for name, v in want.items():
        got = nt.download(name)[: v.size]
        assert np.array_equal(got, v.ravel()), (name, int(np.count_nonzero(got != v.ravel())))
    module.reset_arena()
