"""The cascade's on-chip solves against the oracle's float mirror, bit for bit,
at the sizes where their work splits change: levels of one block, around one
group per warp and one CTA, around a cluster's capacity, odd block counts, and
sparse levels with coarser neighbours, domain faces and the compat quirk."""
import numpy as np
import pytest

from dcgrid_gb300 import capi
from tests import scenarios

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("cuda_ok", "dcg_lib", "oracle_lib")]


def pair(p, noise):
    from dcgrid_gb300 import Simulation
    from oracle.pyoracle import OracleSim
    g, o = Simulation(p), OracleSim(p, precision="float")
    for s in (g, o):
        s.add_velocity_noise(5, noise)
    return g, o


def same(g, o, fields=("pressure", "pressure_tmp", "divergence", "vel_x", "vel_y", "vel_z")):
    alloc = np.repeat(o.get_topology()["pos"][:, 3] >= 0, 64)
    for f in fields:
        a, b = g.get_field(f)[alloc], o.get_field(f)[alloc].astype(np.float32)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), f"{f}: {(a != b).sum()} cells differ"


# (domain, levels, budget of the finest level as a share of its blocks, sweeps);
# blocks of the coarsest level: 1, 3, 63, 64, 65, 130, 1053
SIZES = [
    ((8, 8, 8), 2, 1.0, 4),
    ((24, 8, 8), 2, 0.5, 2),
    ((24, 24, 56), 2, 0.3, 6),
    ((32, 32, 32), 2, 0.5, 6),
    ((40, 104, 8), 2, 0.2, 6),
    ((80, 104, 8), 2, 0.7, 4),
    ((72, 72, 104), 2, 0.25, 4),
    ((64, 48, 80), 3, 0.6, 10),
]


@pytest.mark.parametrize("compat", [0, 1])
@pytest.mark.parametrize("size,levels,share,iters", SIZES)
def test_small_levels_bitexact(size, levels, share, iters, compat):
    gx, gy, gz = size
    full = [(gx >> (l + 2)) * (gy >> (l + 2)) * (gz >> (l + 2)) for l in range(levels)]
    p = scenarios.plume(gx, gy, gz, sum(full[1:]) * 3 // 2 + max(1, int(share * full[0])), levels, iters)
    p.src_radius = min(p.src_radius, min(size) / 4.0)
    p.ref_compat = compat
    g, o = pair(p, 0.5)
    for step in range(2):
        for stage in ("advect_velocity", "adapt", "project", "advect_scalars"):
            getattr(g, stage)()
            getattr(o, stage)()
        g.sync()
        same(g, o)
    for s in (g, o):
        s.project_local()
    g.sync()
    same(g, o)


@pytest.mark.parametrize("scale", [1e-33, 1e-36, 1e-39])
def test_subnormal_pressures_bitexact(scale):
    """Velocities so small, in one corner of a still domain, that the sweeps
    run through subnormal and zero pressures, where the division takes its
    other branches."""
    p = scenarios.plume(32, 64, 32, None, 2, 40)
    g, o = pair(p, 0.0)
    v = np.zeros(g.num_cells, np.float32)
    v[:4096] = scale * np.random.default_rng(3).standard_normal(4096).astype(np.float32)
    for s in (g, o):
        s.set_field("vel_y", v)
        s.project()
    g.sync()
    same(g, o)
