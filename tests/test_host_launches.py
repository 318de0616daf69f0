"""The library's host code (launch attributes, routes, step graphs) on the CPU,
with a runtime that records the launches (tests/fake_gpu.py)."""
import pytest

from dcgrid_gb300 import capi
from tests import scenarios
from tests.fake_gpu import fake, fake_path  # noqa: F401


def dense_scene():
    """two levels in full, the finer one of 40960 blocks"""
    return scenarios.plume(160, 128, 128, 40960 + 5120, 2, 6)


@pytest.mark.parametrize("scene,mode,kernel", [
    (dense_scene, capi.MODE_ADAPTIVE, "k_dense_pass"),
    (lambda: scenarios.plume(32, 32, 32, 64 + 100, 2, 4), capi.MODE_ADAPTIVE, "k_decideILi0E"),
    (lambda: scenarios.ref_default(64, 64, 64, 0), capi.MODE_UNIFORM, "k_u_small"),
    (lambda: scenarios.ref_default(64, 64, 64, 0), capi.MODE_UNIFORM, "k_dense_pass")])
def test_large_shared_memory_on_every_device(fake, scene, mode, kernel):  # noqa: F811
    """The opt-in to large shared memory belongs to the device: a handle on a
    second GPU of the process needs its own."""
    from dcgrid_gb300 import Simulation
    for device in (0, 1):
        fake.device(device)
        s = Simulation(scene(), mode)
        s.step(1)
        s.project()
        assert any(kernel in n for n in fake.launches()), device
