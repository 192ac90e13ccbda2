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
