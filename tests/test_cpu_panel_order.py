"""The cooperative kernels' panels and blocked solves (kern_coop.cu: factor_panels, factor_panels_f32, solve_rows,
solve_rows_f32) give every element the operations of the pivot-by-pivot elimination and of the row-by-row solve
(kin_solver.h:97-139), in that order. Both emulated with exactly rounded FMAs (FP32: rounded again) on random
filled patterns, in the kernels' phases; they must agree bit for bit."""
import random

import numpy as np
import pytest

from test_cpu_elimination_order import filled_pattern, fma, pivot_by_pivot


def f32(v):
    return float(np.float32(v))


def fma32(a, b, c):
    return f32(fma(a, b, c))


def pivots32(a, pat, n, ghinv):
    a = [r[:] for r in a]
    for k in range(n):
        inv = f32(1.0 / f32(a[k][k] + ghinv))
        for i in range(k + 1, n):
            if pat[i][k]:
                l = f32(a[i][k] * inv)
                for j in range(k + 1, n):
                    if pat[k][j]:
                        a[i][j] = fma32(-l, a[k][j], a[i][j])
                a[i][k] = l
        a[k][k] = inv
    return a


def panels(a, pat, n, ghinv, B, single):
    """B pivots per pass: the panel a row at a time, the block's U rows a column at a time, the trailing elements.
    single: FP32, without pattern tests, as an element off the pattern is (plus or minus) zero."""
    mul, f, rnd = (fma32, f32, f32) if single else (fma, float, float)
    a = [r[:] for r in a]
    on = (lambda i, j: True) if single else (lambda i, j: pat[i][j])
    for k in range(0, n, B):
        nb = min(B, n - k)
        j0 = k + nb
        pa = {i: [a[i][k + p] for p in range(nb)] for i in range(k, n)}      # a thread per row
        ux = {j: [a[k + p][j] for p in range(nb)] for j in range(j0, n)}     # a thread per column, loaded ahead
        Lp = {}
        for p in range(nb):
            kp = k + p
            inv = rnd(1.0 / f(pa[kp][p] + ghinv))
            Lp[kp] = pa[kp][:]          # what the pivot row's thread publishes, its own multipliers included
            pa[kp][p] = inv
            for i in range(kp + 1, n):
                if on(i, kp):
                    l = pa[i][p] = rnd(pa[i][p] * inv)
                    for q in range(p + 1, nb):
                        if on(kp, k + q):
                            pa[i][q] = mul(-l, Lp[kp][q], pa[i][q])
        for i in range(k, n):
            a[i][k:j0] = pa[i]
        for j in range(j0, n):
            for p in range(1, nb):
                for q in range(p):
                    if on(k + p, k + q) and on(k + q, j) and on(k + p, j):
                        ux[j][p] = mul(-Lp[k + p][q], ux[j][q], ux[j][p])
            for p in range(nb):
                a[k + p][j] = ux[j][p]
        for i in range(j0, n):
            for j in range(j0, n):
                for p in range(nb):
                    if on(i, k + p) and on(k + p, j):
                        a[i][j] = mul(-pa[i][p], ux[j][p], a[i][j])
    return a


def solve(a, pat, n, b, mul, rnd):
    x = b[:]
    for i in range(n):
        for k in range(i):
            if pat[i][k]:
                x[i] = mul(-a[i][k], x[k], x[i])
    for i in reversed(range(n)):
        for k in reversed(range(i + 1, n)):
            if pat[i][k]:
                x[i] = mul(-a[i][k], x[k], x[i])
        x[i] = rnd(x[i] * a[i][i])
    return x


def blocked_solve(a, pat, n, b, mul, rnd, B, single):
    """Blocks of B columns: their own rows column by column, then the rows past them."""
    on = (lambda i, j: True) if single else (lambda i, j: pat[i][j])
    xi = b[:]          # what each row's thread holds
    for k0 in range(0, n, B):
        end = min(n, k0 + B)
        for k in range(k0, end):
            for i in range(k + 1, end):
                if on(i, k):
                    xi[i] = mul(-a[i][k], xi[k], xi[i])
        for i in range(end, n):
            for k in range(k0, end):
                if on(i, k):
                    xi[i] = mul(-a[i][k], xi[k], xi[i])
    for k0 in reversed(range(0, n, B)):
        end = min(n, k0 + B)
        for k in reversed(range(k0, end)):
            xi[k] = rnd(xi[k] * a[k][k])
            for i in range(k0, k):
                if on(i, k):
                    xi[i] = mul(-a[i][k], xi[k], xi[i])
        for i in range(k0):
            for k in reversed(range(k0, end)):
                if on(i, k):
                    xi[i] = mul(-a[i][k], xi[k], xi[i])
    return xi


def system(rnd, n, single):
    pat = filled_pattern(n, rnd.choice([0.05, 0.2, 0.5, 0.9]), rnd)
    conv = f32 if single else float
    a = [[conv(rnd.uniform(-1, 1) * 10 ** rnd.uniform(-3, 3)) if pat[i][j] else 0.0 for j in range(n)] for i in range(n)]
    b = [conv(rnd.uniform(-1, 1) * 10 ** rnd.uniform(-3, 3)) for _ in range(n)]
    return pat, a, b, conv(10 ** rnd.uniform(0, 4))


@pytest.mark.parametrize("single,B,C", [(False, 4, 8), (True, 8, 32), (True, 8, 4)])
def test_panels_and_solves_same_bits(single, B, C):
    rnd = random.Random(B + C + single)
    for trial in range(25):
        n = rnd.choice([1, 2, 3, 4, 5, 7, 8, 9, 12, 17, 23, 33])
        pat, a, b, ghinv = system(rnd, n, single)
        lu = (pivots32 if single else pivot_by_pivot)(a, pat, n, ghinv)
        got = panels(a, pat, n, ghinv, B, single)
        assert all(got[i][j].hex() == lu[i][j].hex() if pat[i][j] else got[i][j] == 0.0 for i in range(n) for j in range(n)), (trial, n)
        mul, conv = (fma32, f32) if single else (fma, float)
        x, y = solve(lu, pat, n, b, mul, conv), blocked_solve(lu, pat, n, b, mul, conv, C, single)
        assert [v.hex() for v in x] == [v.hex() for v in y], (trial, n)
