"""The lane-group kernels' schedule image (kin_mech_group_image): every element of the RHS, the
Jacobian and the elimination is listed with the operations of the reference's table walk
(src/sim/kinetics/kin_solver.h:40-139) in its order, and every index stays inside its array."""
import ctypes as C

import numpy as np
import pytest

import simstack_gb300 as sg

NONE = 0xFFFF
FIELDS = ("n R ld pairs rx pr fround forder jrounds jround jdst nzero zero pivot mask rr pfirst pidx words odd").split()


def image(km, lanes, prec):
    L = sg.lib()
    size = L.kin_mech_group_image(C.byref(km), lanes, prec, None, 0)
    buf = np.zeros(size // 4, np.uint32)
    assert L.kin_mech_group_image(C.byref(km), lanes, prec, buf.ctypes.data, size) == size
    return buf.astype(np.int64), dict(zip(FIELDS, (int(v) for v in buf[: len(FIELDS)])))


def mechanisms():
    yield "air", sg.Model.air()
    for n, R, seed in ((3, 6, 2), (8, 24, 7), (16, 48, 5), (20, 40, 1), (24, 80, 5), (32, 64, 1), (32, 48, 2)):
        yield f"{n}x{R}", sg.Model.synthetic(seed=seed, species=n, reactions=R, bimolecular=0.7, products=1)


def coefficient(word, prec):
    top = int(word) >> 16
    if prec == 0:
        return float(np.array([top << 48], np.uint64).view(np.float64)[0])
    return float(np.array([top << 16], np.uint32).view(np.float32)[0])


def gathered(w, h, first, dst, rounds, lanes, prec, none):
    """{target: [(offset, coefficient)]} of a gather's rounds."""
    out = {}
    for q in range(rounds):
        off, length = w[first + 2 * q], w[first + 2 * q + 1]
        assert off + (length + 8) * lanes <= h["words"]   # the kernels read a batch ahead
        for lane in range(lanes):
            words = [w[off + e * lanes + lane] for e in range(length)]
            terms = [((int(v) & 0x7FFF), coefficient(v, prec)) for v in words]
            live = [t for t in terms if t[0] != none]
            assert terms[: len(live)] == live and all(c == 0.0 and np.signbit(c) for _, c in terms[len(live):])
            to = w[dst + q * lanes + lane]
            if to == NONE:
                assert not live
            else:
                out[int(to)] = live
    return out


@pytest.mark.parametrize("prec", [0, 1, 4])
@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_schedule_lists_the_table_walk(lanes, prec):
    for name, model in mechanisms():
        km = model.kinmech()
        w, h = image(km, lanes, prec)
        n, R, ld = h["n"], h["R"], h["ld"]
        rate, lu = (4 if prec == 1 else 8), (8 if prec == 0 else 4)
        rx = [km.reactions[r] for r in range(R)]
        reac = [list(x.reactant[: x.reactant_count]) for x in rx]
        # rates and the Jacobian's products
        got = {int(v) & 255: [(int(v) >> (8 + 6 * p)) & 63 for p in range(int(v) >> 26)] for v in w[h["rx"]:h["rx"] + R]}
        assert got == dict(enumerate(reac)), name
        pair = {}
        for r in range(R):
            for p in range(len(reac[r])):
                q = int(w[h["pidx"] + w[h["pfirst"] + r] + p])
                v = int(w[h["pr"] + q])
                assert v & 255 == r and [(v >> (8 + 6 * c)) & 63 for c in range(v >> 26)] == reac[r][:p] + reac[r][p + 1:]
                pair[r, p] = q
        assert sorted(pair.values()) == list(range(h["pairs"]))
        # RHS and -J: terms per species / entry, in the table walk's order
        want = {s: [] for s in range(n)}
        jac = {}
        for r in range(R):
            for e in range(rx[r].net_count):
                want[rx[r].net_species[e]].append((r * rate, float(rx[r].net_coef[e])))
            for p in range(len(reac[r])):
                for e in range(rx[r].net_count):
                    at = (rx[r].net_species[e] * ld + reac[r][p]) * lu
                    jac.setdefault(at, []).append((pair[r, p] * lu, -float(rx[r].net_coef[e])))
        assert gathered(w, h, h["fround"], h["forder"], -(-n // lanes), lanes, prec, R * rate) == want, name
        assert gathered(w, h, h["jround"], h["jdst"], h["jrounds"], lanes, prec, h["pairs"] * lu) == jac, name
        # the filled pattern, the fill-in that starts at zero, and the updates of every element by pivot
        pat = np.eye(n, dtype=bool)
        for i in range(n):
            for lst, beg in ((km.lower, km.lower_begin), (km.upper, km.upper_begin)):
                for e in range(beg[i], beg[i + 1]):
                    pat[i, lst[e].col] = True
        zero = {int(v) for v in w[h["zero"]:h["zero"] + h["nzero"]]}
        assert zero == {(i * ld + j) * lu for i in range(n) for j in range(n) if pat[i, j]} - set(jac), name
        for k in range(n):
            rows, nr, tasks, nt = (int(v) for v in w[h["pivot"] + 4 * k:h["pivot"] + 4 * k + 4])
            assert nr % lanes == 0 and nt % lanes == 0
            spare = n * ld * lu
            below = [int(v) for v in w[rows:rows + nr] if v != spare]
            assert below == [i * ld * lu for i in range(k + 1, n) if pat[i, k]], name
            done = []
            for v in w[tasks:tasks + nt]:
                ij, i0 = int(v) & 0xFFFF, int(v) >> 16
                j = (ij - i0) // lu
                assert i0 % (ld * lu) == 0 and 0 <= j < n and ij < (n + 1) * ld * lu
                if i0 != spare:
                    done.append((i0 // (ld * lu), j))
            assert done == [(i, j) for i in range(k + 1, n) for j in range(k + 1, n) if pat[i, k] and pat[k, j]], name
        for i in range(n):
            lo, hi = (int(v) for v in w[h["mask"] + 2 * i:h["mask"] + 2 * i + 2])
            assert [j for j in range(n) if (lo | hi) >> j & 1] == [j for j in range(n) if j != i and pat[i, j]]
            assert lo >> i == 0 and hi & ((2 << i) - 1) == 0


def test_record_that_is_not_the_symbolic_phases_gets_no_image():
    """Valid tables whose lists are in another order or miss an update keep to the table walk."""
    base = sg.Model.air().kinmech()

    def size(km):
        return sg.lib().kin_mech_group_image(C.byref(km), 8, 0, None, 0)

    def changed(edit):
        km = sg.KinMech.from_buffer_copy(sg.kinmech_bytes(base))
        edit(km)
        return km

    def swap_lower(km):
        i = next(i for i in range(17) if km.lower_begin[i + 1] - km.lower_begin[i] > 1)
        a, b = km.lower[km.lower_begin[i]], km.lower[km.lower_begin[i] + 1]
        (a.index, a.col), (b.index, b.col) = (b.index, b.col), (a.index, a.col)

    def drop_update(km):
        d = next(d for d in range(km.lu_div_count) if km.lu_div[d].sub_end > km.lu_div[d].sub_begin)
        km.lu_div[d].sub_end -= 1

    def other_slot(km):
        km.reactions[0].jac_index[0][0] = km.diag[16]

    assert size(base) > 0
    for edit in (swap_lower, drop_update, other_slot):
        assert size(changed(edit)) == 0, edit.__name__
