"""The module's host code on a stand-in runtime (fake_runtime.py): what it launches, keeps and answers when a
device call fails or an optional resource is missing."""
import numpy as np
import pytest

import simstack_gb300 as sg

from fake_runtime import Fake


@pytest.fixture
def fake(monkeypatch):
    return Fake(monkeypatch)


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
