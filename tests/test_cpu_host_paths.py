"""The module's host code on a stand-in runtime (fake_runtime.py): what it launches, keeps and answers when a
device call fails or an optional resource is missing."""
import numpy as np
import pytest

import simstack_gb300 as sg

from fake_runtime import Fake


@pytest.fixture
def fake(monkeypatch):
    f = Fake(monkeypatch)
    yield f
    f.module.set_straggler_budget(sg.DEFAULT_STRAGGLER_BUDGET)   # what gpu_init leaves as it is
    sg.check(sg.lib().gpu_kin_set_straggler_block(128), "gpu_kin_set_straggler_block")


def advanced(fake, cells=100, precision=0, **kw):
    """The kernels of an advance of `cells` air cells."""
    fake.launches()
    fake.module.reset_arena()
    fake.module.integrate(sg.air_cells(cells, seed=1), 1.0, precision=precision, **kw)
    return fake.launches()


def test_images_that_found_no_memory_are_tried_again(fake):
    """The same record set again, with memory at hand, gets its group kernels."""
    km = sg.Model.air().kinmech()
    fake.fail("cudaMalloc")
    fake.module.set_mech(km)
    assert "kin_group_kernel" not in advanced(fake)[0]["name"]
    fake.module.set_mech(km)
    assert "kin_group_kernel" in advanced(fake)[0]["name"]


def test_f32_lanes_past_one_wave_run_the_queue(fake):
    """The static kernel does not refill a lane whose cell is done: it takes batches whose cells are all on the GPU."""
    fake.module.set_mech(sg.Model.air().kinmech())
    for cells, kernel in ((64, "kin_static_kernel"), (152 * 256, "kin_static_kernel"), (152 * 256 + 8, "kin_queue_cta_kernel")):
        assert [kernel in k["name"] for k in advanced(fake, cells=cells, precision=1)] == [True], cells


@pytest.mark.parametrize("precision,per_sm,group", [(0, 64, True), (0, 65, False), (2, 34, True), (2, 36, False), (2, 35, False)])
def test_groups_end_where_they_fill_the_gpu_once(fake, precision, per_sm, group):
    fake.module.set_mech(sg.Model.air().kinmech())
    assert ("kin_group_kernel" in advanced(fake, cells=152 * per_sm, precision=precision)[0]["name"]) == group


@pytest.mark.parametrize("precision,species,per_sm,group,drain", [
    (0, 3, 40, True, 0), (0, 3, 100, False, 0), (0, 8, 110, True, 0), (0, 8, 197, False, 0), (0, 16, 390, True, 0), (0, 16, 431, False, 0),
    (1, 1, 20, True, 0), (1, 3, 145, True, 0), (1, 3, 431, False, 0), (1, 6, 990, False, 0), (1, 16, 990, True, 0),
    (2, 1, 98, False, 0), (2, 2, 70, True, 0), (2, 2, 197, False, 16), (2, 3, 431, False, 16), (2, 8, 990, True, 0)])
def test_table_mechanisms_go_where_they_are_faster(fake, precision, species, per_sm, group, drain):
    """A few species' lanes beat the groups from far smaller batches on, and a CTA of them parks few of its cells."""
    if species > 1:
        m = sg.Model.synthetic(seed=5, species=species, reactions=2 * species)
    else:
        m = sg.Model.new()
        m.add_species("S0", True)
        m.add_reaction("S0 -> S0 + S0")
        m.finalize()
        m.k_const = np.array([0.7])
    fake.module.set_mech(m.kinmech())
    fake.launches()
    fake.module.integrate(sg.synthetic_cells(m, 152 * per_sm, seed=1), 1.0, precision=precision)
    first, *rest = fake.launches()
    assert ("kin_group_kernel" in first["name"]) == group and first["drain"] == drain
    assert len(rest) == (0 if group or precision == 1 else 1)   # the hand-off's


@pytest.mark.parametrize("precision,cells,chunks,kernel,block", [
    (2, 50000, 4, "kin_queue_cta_kernel", 128), (2, 50000, 2, "kin_queue_cta_kernel", 256), (2, 50000, 1, "kin_queue_cta_kernel", 256),
    (2, 5000, 4, "kin_group_kernel", None), (1, 50000, 4, "kin_static_kernel", 64), (1, 50000, 2, "kin_queue_cta_kernel", 128)])
def test_pipelined_chunks_take_a_chunks_shape(fake, precision, cells, chunks, kernel, block):
    """What a lane kernel has to do is its chunk, not the batch."""
    fake.module.set_mech(sg.Model.air().kinmech())
    fake.launches()
    fake.module.integrate_pipelined(sg.air_cells(cells, seed=1), 1.0, precision=precision, chunks=chunks)
    launched = fake.launches()
    assert len(launched) == chunks
    assert all(kernel in k["name"] and (block is None or k["block"] == block) for k in launched)


@pytest.mark.parametrize("groups,cells,substeps,resident", [
    (200, 240, 1, False), (200, 240, 23, False), (200, 240, 24, True), (64, 100, 31, False), (64, 100, 32, True), (64, 2304, 11, False),
    (64, 2304, 12, True), (200, 1, 253, False), (1, 100, 15, False), (1, 100, 16, True), (1, 240, 6, True), (1, 999, 2, False),
    (1, 999, 3, True), (1, 1000, 0, False), (1, 1000, 1, True), (64, 240, 253, True), (1, 2305, 253, False)])
def test_film_windows_of_few_substeps_run_through_memory(fake, groups, cells, substeps, resident):
    """The resident kernel's loads, stores and evaporation sum want some substeps to pay for them."""
    sites = cells // 3
    nt = sg.NftTransport(fake.module, groups, cells, sites, 1, 3)
    nt.run(np.ones(9), 24.0, 150.0, 900.0, 140.0, substeps)
    (k,) = fake.launches()
    assert ("nft_resident_kernel" in k["name"]) == resident


def reordered(km):
    """The record with two entries of a row's lower list in the other order: valid, but without group images."""
    km = sg.KinMech.from_buffer_copy(sg.kinmech_bytes(km))
    i = next(i for i in range(17) if km.lower_begin[i + 1] - km.lower_begin[i] > 1)
    a, b = km.lower[km.lower_begin[i]], km.lower[km.lower_begin[i] + 1]
    (a.index, a.col), (b.index, b.col) = (b.index, b.col), (a.index, a.col)
    return km


def test_stragglers_without_group_images_go_to_the_cooperative_kernel(fake):
    fake.module.set_mech(reordered(sg.Model.air().kinmech()))
    sg.check(sg.lib().gpu_kin_set_straggler_block(64), "gpu_kin_set_straggler_block")
    lanes, rest = advanced(fake)
    assert "kin_queue_cta_kernel" in lanes["name"] and lanes["budget"] > 0 and lanes["drain"] == 0
    assert "kin_coop_kernel<0>" in rest["name"] and rest["resume"] == 1 and rest["block"] == 64
    assert len(advanced(fake, precision=2)) == 1   # mixed cells stay on their lanes
    fake.module.set_straggler_budget(0)
    assert len(advanced(fake)) == 1


def test_a_failed_set_mech_leaves_no_other_mechanisms_tables(fake):
    """Images that could not be written: the cooperative shape has nothing to run on and says so."""
    small = sg.Model.synthetic(seed=2, species=3, reactions=6)
    fake.module.set_mech(small.kinmech())
    fake.module.set_tuning(kind=3, block=32)
    fake.fail("cudaMemcpy", error=999)
    with pytest.raises(sg.GpuError):
        fake.module.set_mech(sg.Model.air().kinmech())
    with pytest.raises(sg.GpuError):
        fake.module.integrate(sg.air_cells(8, seed=1), 1.0)
    assert fake.launches() == []


@pytest.mark.parametrize("precision", [0, 2])
def test_parked_cells_are_the_last_advances(fake, precision):
    """A batch on the group kernels parks nothing, whatever the batch before it parked."""
    fake.module.set_mech(sg.Model.air().kinmech())
    fake.L.fake_park(7)
    lanes, rest = advanced(fake, cells=20000, precision=precision)
    assert "kin_queue_cta_kernel" in lanes["name"] and rest["resume"] == 1
    assert fake.module.parked_cells() == 7
    assert len(advanced(fake, precision=precision)) == 1
    assert fake.module.parked_cells() == 0


@pytest.mark.parametrize("precision", [0, 2])
def test_parked_cells_are_finished_whatever_the_wait_limit(fake, precision):
    """The limit of the table-staging waits ends the lane kernel before it steps a cell; cells that it parked have been
    stepped, and are not left half-way."""
    m = sg.Model.synthetic(seed=5, species=8, reactions=24)
    fake.module.set_mech(m.kinmech())
    fake.module.set_tuning(kind=2)
    fake.launches()
    sg.check(sg.lib().gpu_kin_set_wait_limit(1), "gpu_kin_set_wait_limit")
    fake.module.integrate(sg.synthetic_cells(m, 500, seed=1), 1.0, precision=precision)
    sg.check(sg.lib().gpu_kin_set_wait_limit(1 << 24), "gpu_kin_set_wait_limit")
    lanes, rest = fake.launches()
    assert lanes["wait_polls"] == 1 and rest["resume"] == 1 and rest["wait_polls"] > 1 << 20


CELLS = 64000   # lanes: past the group kernels' sizes, each CTA parks what it has left


@pytest.fixture
def serving(fake):
    """A table mechanism of three species (184 bytes a cell), mixed, and the budget of one request."""
    m = sg.Model.synthetic(seed=2, species=3, reactions=6)
    base = 8 * (3 * 3 + 6 + 8) * CELLS + 8 * 3
    opened = []

    def run(budget, requests):
        s = sg.Server(budget)
        opened.append(s)
        s.set_mech(m.kinmech())
        y, k = np.full((3, CELLS), 1e-6), np.repeat(m.k_const[:, None], CELLS, 1)
        for _ in range(requests):
            s.submit(y, k, 1, 64, 0.05, mechanism=1, precision=2)
        running = s.progress()[0]
        return s.stats(), running, fake.stream_bytes(), fake.launches()

    run.one = base + 256 + table_bytes(fake)
    yield run
    for s in opened:
        s.close()


def table_bytes(fake):
    """A request's table image: the smallest budget that takes a request of one cell tells it."""
    s = sg.Server(1 << 30)
    s.submit(np.full((17, 8), 1e10), np.full((44, 8), 1e-10), 1, 8, 0.05)
    s.progress()
    n = s.stats()["in_use_bytes"] - 8 * (3 * 17 + 44 + 8) * 8 - 8 * 17 - 256
    s.close()
    fake.launches()
    return n


def test_served_hand_off_is_inside_the_budget(serving):
    stats, running, (now, peak), launches = serving(1 << 30, 1)
    assert running == 1 and any(k["resume"] for k in launches)
    assert now <= stats["in_use_bytes"] and peak <= stats["peak_bytes"]


def test_served_request_that_fills_the_budget_keeps_its_cells(serving):
    stats, running, (now, _), launches = serving(serving.one, 1)
    assert running == 1 and not any(k["resume"] for k in launches)
    assert now == stats["in_use_bytes"] == serving.one


@pytest.mark.parametrize("spare", [0, 100000])
def test_served_hand_off_keeps_no_request_waiting(serving, spare):
    stats, running, (now, _), _ = serving(2 * serving.one + spare, 2)
    assert running == 2 and now <= stats["in_use_bytes"] <= stats["budget_bytes"]


def test_a_failed_serve_set_mech_keeps_the_mechanism_before(fake):
    """A request's arrays are read by the species and reactions of the mechanism that is in force."""
    old, new = sg.Model.synthetic(seed=2, species=3, reactions=6), sg.Model.synthetic(seed=7, species=8, reactions=24)
    y, k = np.full((3, 8), 1e-6), np.repeat(old.k_const[:, None], 8, 1)
    with sg.Server(1 << 30) as s:
        s.set_mech(old.kinmech())
        s.submit(y, k, 1, 8, 0.05, mechanism=1)
        s.progress()
        one = s.stats()["in_use_bytes"]
        s.drain()
        fake.fail("cudaMemcpy", error=999)
        with pytest.raises(sg.GpuError):
            s.set_mech(new.kinmech())
        rid = s.submit(y, k, 1, 8, 0.05, mechanism=1)
        s.progress()
        assert s.poll(rid)["state"] == "running" and s.stats()["in_use_bytes"] == one
