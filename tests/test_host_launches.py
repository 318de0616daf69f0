"""The library's host code (launch attributes, routes, step graphs) on the CPU,
with a runtime that records the launches (tests/fake_gpu.py)."""
import numpy as np
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


def small_scene():
    return scenarios.plume(32, 32, 32, None, 2, 4)


@pytest.mark.parametrize("batch", [False, True])
def test_refused_launch_leaves_no_step_graph(fake, batch):  # noqa: F811
    """A launch that the device refuses has no node in the graph under capture:
    every step reports it, none is replayed without it, and the state is the one
    before the step."""
    from dcgrid_gb300 import Batch, DcgError, Simulation

    def handle():
        h = Batch([small_scene(), small_scene()]) if batch else Simulation(small_scene())
        return h, (h[0] if batch else h)
    h, sim = handle()
    velocity = np.arange(sim.num_cells, dtype=np.float32)
    sim.set_field("vel_x", velocity)
    fake.refuse("k_cluster_solve")
    fake.launches()
    for capture in (True, True, True, False):
        if not capture:  # the legacy stream cannot be captured
            fake.refuse("")
            h.set_stream(0)
        with pytest.raises(DcgError) as e:
            h.step(1)
        assert e.value.code == capi.DCG_E_CUDA
        assert fake.launches() == []
        assert np.array_equal(sim.get_field("vel_x"), velocity)
    assert sim.stats().steps == 0
    h.set_stream(1)
    fake.launches()
    h.step(2)
    got = fake.launches()
    assert any("k_cluster_solve" in n for n in got)
    fresh = handle()[0]
    fake.launches()
    fresh.step(2)
    assert got == fake.launches()


def test_partly_allocated_full_level_is_solved(fake):  # noqa: F811
    """A topology from outside may hold fewer blocks of a level than its budget,
    which covers the block grid: the device counts them, so the cluster solve has
    to be launched over that level as over a sparse one."""
    from dcgrid_gb300 import Simulation
    s = Simulation(scenarios.plume(64, 64, 64, 512 + 4096, 2, 4))
    assert s.info.budget[0] == s.info.full_blocks[0] == 4096  # more than a cluster holds
    fake.launches()
    s.project()
    assert [n.split(":")[1] for n in fake.launches() if "k_cluster_solve" in n] == ["1-1"]
    fake.raster_bad(True)
    s.set_topology(s.get_topology())
    fake.launches()
    s.project()
    assert [n.split(":")[1] for n in fake.launches() if "k_cluster_solve" in n] == ["1-0"]


@pytest.mark.parametrize("sms,blocks,solver", [(152, (32, 32, 38), "k_resident_solve"), (152, (33, 33, 36), "k_dense_pass"),
                                               (148, (32, 32, 37), "k_resident_solve"), (148, (34, 34, 33), "k_dense_pass")])
def test_full_levels_beyond_the_resident_solve_are_dense(fake, sms, blocks, solver):  # noqa: F811
    """The resident solve holds 256 blocks per SM; a full level of one more goes
    to the dense passes, whatever the number of SMs, and none to the general solve."""
    from dcgrid_gb300 import Simulation
    fake.sms(sms)
    x, y, z = blocks
    s = Simulation(scenarios.plume(4 * x, 4 * y, 4 * z, x * y * z, 1, 4))
    fake.launches()
    s.project()
    names = fake.launches()
    used = {k for k in ("k_resident_solve", "k_dense_pass", "k_level_solve_batch") if any(k in n for n in names)}
    assert used == {solver}


def test_autotune_does_not_rank_a_general_solve_without_work(fake):  # noqa: F811
    """Levels that the clusters hold never reach the general solve: its variants
    have nothing to do, and their times would be noise."""
    from dcgrid_gb300 import Batch
    fake.cost("k_level_solve_batchILi8E", 1e-6)
    fake.cost("k_cluster_solve", 0.05)
    b = Batch(scenarios.plume_batch(3, 17, sizes=(16, 32), iters=10))
    fake.launches()
    t = b.autotune(spinup_steps=0, reps=1)
    assert not any("k_level_solve_batch" in n for n in fake.launches())
    assert (t["solve_cache"], t["solve_ctas_per_sm"]) == (19, 0)
    assert t["solve_ms"] == pytest.approx(0.05)


def test_autotune_times_the_general_solve_itself(fake):  # noqa: F811
    """Levels that the resident solve takes while few of their blocks are
    allocated, and the general solve afterwards: the latter is timed with work,
    the cheapest of its variants chosen."""
    from dcgrid_gb300 import Batch
    fake.cost("k_level_solve_batch", 1.0)
    fake.cost("k_level_solve_batchILi2ELi3E", 0.5)  # variant 34
    fake.load(30000)
    b = Batch([scenarios.plume(160, 160, 128, 6400 + 46601, 2, 4)])
    fake.launches()
    t = b.autotune(spinup_steps=1, reps=1)
    timed = [n for n in fake.launches() if "k_level_solve_batch" in n and n.endswith("<0")]
    assert t["solve_cache"] == 34 and len(timed) > 13


def test_kernels_write_only_buffers_that_a_copy_would_take(fake):  # noqa: F811
    """A 16-bit field widens straight into an aligned buffer of the handle's GPU
    that holds all of it. Anything else goes through a copy, which takes any
    address and refuses one that runs past its allocation."""
    import ctypes as C
    from dcgrid_gb300 import Simulation
    p = small_scene()
    p.precision = capi.PRECISION_MIXED_FP16
    s = Simulation(p)
    n = 4 * s.num_cells

    def into(buffer, offset=0):
        """(status, whether a copy wrote the buffer); the kernels do nothing here"""
        C.memset(buffer, 7, n // 2)
        rc = s.L.dcg_get_field(s.h, capi.FIELD_NAMES["density"], C.c_void_p(buffer + offset), capi.DEVICE)
        return rc, C.string_at(buffer + offset, n // 2 - offset) != b"\7" * (n // 2 - offset)
    own = fake.malloc(n + 8)
    assert into(own) == (capi.DCG_OK, False)
    assert into(own, 4) == (capi.DCG_OK, False)
    assert into(own, 2) == (capi.DCG_OK, True)
    small = fake.malloc(n // 2)
    fake.malloc(n)
    assert into(small) == (capi.DCG_E_CUDA, False)
    fake.lib.cudaGetLastError()
    fake.device(1)
    other = fake.malloc(n)
    fake.device(0)
    assert into(other) == (capi.DCG_OK, True)


def test_frame_scratch_is_counted(fake):  # noqa: F811
    """device_bytes is the memory that the handle holds, a frame's tiles and map
    (allocated by the first frame) included; none of it is left behind."""
    import ctypes as C
    from dcgrid_gb300 import Simulation
    from dcgrid_gb300.sim import default_render_params
    held = fake.held()
    p = small_scene()
    s = Simulation(p)
    before = s.info.device_bytes
    assert fake.held() - held == before
    rp = default_render_params(8, 8, p)
    image = fake.malloc(8 * 8 * 16)
    for _ in range(2):
        assert s.L.dcg_render(s.h, C.byref(rp), C.c_void_p(image), capi.DEVICE) == capi.DCG_OK
        s.L.dcg_get_info(s.h, C.byref(s.info))
        assert s.info.device_bytes == fake.held() - held - 8 * 8 * 16 > before
    s.close()
    assert fake.held() - held == 8 * 8 * 16


def test_a_solver_that_gives_way_hides_no_other_refusal(fake):  # noqa: F811
    """The resident solve, when refused, leaves its levels to the general solve and
    no error; an error that is there already stays."""
    from dcgrid_gb300 import DcgError, Simulation
    s = Simulation(scenarios.plume(64, 64, 64, 512 + 4000, 2, 4))
    fake.refuse("k_resident_solve")
    fake.launches()
    s.step(2)
    assert any("k_level_solve_batch" in n for n in fake.launches())
    s = Simulation(scenarios.plume(64, 64, 64, 512 + 4000, 2, 4))
    fake.refuse("k_decide")
    for _ in range(2):
        with pytest.raises(DcgError):
            s.step(1)
