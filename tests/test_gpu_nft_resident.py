"""The register-resident film kernel against the reference's transport restated per element in numpy f32
(src/sim/nft.cpp:1028-1106: the same operations in the same order, fused steps exact through f64 and one
rounding of their own), at the sizes where its shape changes: one cell, a lane's run, one warp and
several warps per channel, and a channel too long for it."""
import numpy as np
import pytest

import simstack_gb300 as sg

pytestmark = pytest.mark.gpu

REF = np.array([20.0, 8.0, 150.0, 10.0, 40.0, 200.0, 160.0, 50.0, 60.0], np.float32)
ENV = tuple(np.float32(v) for v in (24.0, 150.0, 900.0, 140.0))


def round_odd_sum(p, c):
    """p + c in f64 rounded to odd, so that the following rounding to f32 is the exact sum's."""
    s = p + c
    bb = s - p
    err = (p - (s - bb)) + (c - bb)
    bits = s.view(np.int64)
    away = (err > 0) == (s > 0)
    fix = (err != 0) & (bits & 1 == 0)
    return np.where(fix, np.where(away, bits + 1, bits - 1), bits).view(np.float64)


def fma(a, b, c):
    p = np.ascontiguousarray(a, np.float64) * np.asarray(b, np.float64)   # exact: 48 bits
    return round_odd_sum(p, np.broadcast_to(np.asarray(c, np.float64), p.shape).copy()).astype(np.float32)


def expected(a, cells, sites, offset, stride, substeps):
    x, hot, cold = a["rows"].copy(), a["hot"].copy(), a["cold"]
    site = a["sites"].copy()
    T_amb, radiant, e0, slope = ENV
    kw, kr, ge, ev = (cold[:, :, o:o + 8] for o in (24, 32, 40, 48))
    kT = fma(ge, slope, kw)
    bT = fma(-ge, e0, fma(kw, T_amb - REF[0], kr * radiant))
    hot[:, :, 1], hot[:, :, 2] = kT, bT
    c, ko = hot[:, :, 0], hot[:, :, 3]
    on = offset + np.arange(sites) * stride if sites and offset + (sites - 1) * stride < cells else None
    out = np.zeros_like(x[:, 0])
    s0, s1, s2, s3 = (np.float32(v) for v in (-0.000077774, 0.007991, -0.41022, 14.652))
    for _ in range(substeps):
        out = out + x[:, -1]
        up = np.concatenate([np.zeros_like(x[:, :1]), x[:, :-1]], 1)
        x = fma(c[:, :, None], up - x, x)
        x[:, :, 0] = fma(-kT, x[:, :, 0], x[:, :, 0]) + bT
        A = REF[0] + x[:, :, 0]
        sat = fma(fma(fma(s0, A, s1), A, s2), A, s3)
        x[:, :, 1] = fma(ko, sat - (REF[1] + x[:, :, 1]), x[:, :, 1])
        if on is not None:
            before = x[:, on, 1:].copy()
            t = before - site[:, :, 24:88].reshape(-1, sites, 8, 8)
            after = np.where(t > -REF[1:, None], t, -REF[1:, None])
            x[:, on, 1:] = after
            site[:, :, 224:288] = (site[:, :, 224:288].reshape(-1, sites, 8, 8) + (before - after)).reshape(-1, sites, 64)
    e = np.zeros_like(x[:, 0, 0])
    for j in range(cells):
        e = fma(ev[:, j], fma(np.broadcast_to(slope, e.shape), x[:, j, 0], e0), e)
    return {"rows": x, "hot": hot, "sites": site, "out_sum": out, "evap_kg": e * np.float32(substeps)}


@pytest.mark.parametrize("cells,sites,offset,stride", [(1, 1, 0, 3), (2, 0, 0, 1), (33, 33, 0, 1), (64, 21, 1, 3), (97, 1, 40, 0),
                                                       (240, 80, 1, 3), (241, 61, 0, 4), (301, 43, 5, 7), (700, 10, 690, 1),
                                                       (769, 256, 1, 3), (2304, 2304, 0, 1), (2305, 700, 2, 3), (65, 30, 5, 3)])
def test_shapes_match_the_reference_operations(module, cells, sites, offset, stride):
    rng = np.random.default_rng(cells)
    groups, substeps = 3, 7
    a = {"rows": rng.normal(0.0, 0.5, (groups, cells, 9, 8)).astype(np.float32), "hot": np.zeros((groups, cells, 4, 8), np.float32),
         "cold": np.zeros((groups, cells, 80), np.float32), "sites": np.zeros((groups, sites, 288), np.float32)}
    a["hot"][:, :, 0] = rng.uniform(0.05, 0.9, (groups, cells, 8))
    a["hot"][:, :, 3] = rng.uniform(0.0, 0.02, (groups, cells, 8))
    for off, hi in ((24, 1e-3), (32, 1e-5), (40, 1e-6), (48, 1e-9)):
        a["cold"][:, :, off:off + 8] = rng.uniform(0.0, hi, (groups, cells, 8))
    a["sites"][:, :, 24:88] = rng.uniform(0.0, 30.0, (groups, sites, 64))   # some uptakes reach the floor
    nt = sg.NftTransport(module, groups, cells, sites, offset, stride)
    for name, v in a.items():
        if v.size:
            nt.upload(name, v.ravel())
    nt.run(REF, *ENV, substeps, flush_denormals=False)
    want = expected(a, cells, sites, offset, stride, substeps)
    for name, v in want.items():
        got = nt.download(name)[: v.size]
        assert np.array_equal(got, v.ravel()), (name, int(np.count_nonzero(got != v.ravel())))
    module.reset_arena()
