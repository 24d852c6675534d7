"""Whole runs of steps of a small grid in one launch against a launch per stage.

With the tensor memory off a step is a launch per stage.  Both do the same
operations on every line in the same order, so the tolerance is zero bits,
NaNs included.
"""
import numpy as np
import pytest

from bfvm import Microenvironment
from bfvm import workloads as W

pytestmark = pytest.mark.gpu


def _run(wl, field, tmem, precision, chain, active, steps, plane=False, nodes=None):
    me = Microenvironment.from_workload(wl, precision=precision, upload=False)
    me.set_dirichlet_activation(active)
    me.upload_field(field)
    me.set_fp64_chain(chain)
    me.set_sweep_tmem(tmem)
    if nodes is not None:
        me.set_dirichlet_nodes(*nodes)
    for n in steps:
        if plane:
            me.simulate_diffusion_decay_2d(n, sources=True)
        else:
            me.simulate_diffusion_decay(n, sources=True)
    out = me.download_field()
    me.close()
    return out


# Line lengths about the batches of 16 values and the 8, 16 and 32 lanes of an
# x row; last tiles of one line; face rows only (ny or nz of 1 and 2) and face
# rows past 128 values; one tile and more than 148; eight warps to an SM, and
# the first sizes past that; agents alone, many to a tile (more than 32), so
# many that they go ahead of the sweep, and stacked in a voxel.
SHAPES = [(3, 3, 3, 1, 9), (16, 16, 15, 2, 40), (18, 9, 12, 2, 2000), (17, 33, 31, 3, 3000), (31, 32, 48, 2, 500), (33, 47, 61, 7, 900),
          (64, 64, 64, 9, 2000), (65, 1, 40, 2, 70), (1, 70, 33, 2, 60), (40, 2, 2, 2, 30), (200, 40, 33, 2, 4000),
          (129, 50, 7, 2, 100), (30, 300, 9, 1, 100), (100, 100, 96, 3, 2000)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision,chain", [("fp64", 0), ("fp64", 1), ("fp64", 2), ("fp32", 0), ("fp32", 1)])
def test_resident_steps_equal_a_launch_per_stage(shape, precision, chain):
    nx, ny, nz, S, agents = shape
    wl = W.small_random(9000 + nx + ny + nz, nx=nx, ny=ny, nz=nz, S=S, n_agents=agents, steps=3)
    for active in (np.ones(S, np.uint8), np.arange(S, dtype=np.uint8) % 2):
        a, b = (_run(wl, wl.field0, tmem, precision, chain, active, (1, 4)) for tmem in (1, 0))
        assert np.array_equal(a, b), (shape, precision, chain, active)


@pytest.mark.parametrize("shape", [(1, 40, 1, 1, 20), (33, 16, 1, 2, 300), (80, 33, 1, 2, 9000), (90, 127, 1, 4, 500), (300, 61, 1, 2, 4000)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_resident_plane_steps_equal_a_launch_per_stage(shape, precision):
    nx, ny, nz, S, agents = shape
    wl = W.small_random(77 + nx, nx=nx, ny=ny, nz=nz, S=S, n_agents=agents, steps=3)
    rng = np.random.default_rng(nx)
    m = max(2, nx * ny // 9)
    nodes = (rng.choice(nx * ny, m, replace=False).astype(np.int32), rng.random((m, S)),
             rng.integers(0, 2, (m, S)).astype(np.uint8))
    for nd in (None, nodes):
        a, b = (_run(wl, wl.field0, tmem, precision, 0, np.zeros(S, np.uint8), (1, 3), plane=True, nodes=nd)
                for tmem in (1, 0))
        assert np.array_equal(a, b), (shape, precision, nd is None)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_resident_steps_special_values_and_long_runs(precision):
    """Inputs that the exactness screen sends back, infinities and NaNs; and a
    run of more steps than one launch takes."""
    wl = W.small_random(3, nx=36, ny=30, nz=27, S=2, n_agents=200, steps=2)
    active = np.array([0, 1], np.uint8)
    a, b = (_run(wl, wl.field0, tmem, precision, 0, active, (131,)) for tmem in (1, 0))
    assert np.array_equal(a, b)
    rng = np.random.default_rng(5)
    f = wl.field0.copy()
    odd = [-1.0, 0.0, -0.0, 5e-324, 2.0 ** -960, 2.0 ** -961, -2.0 ** -970, 1e30]
    f[rng.integers(0, f.size, f.size // 50)] = rng.choice(odd, f.size // 50)
    a, b = (_run(wl, f, tmem, precision, 0, active, (2,)) for tmem in (1, 0))
    assert np.array_equal(a, b)
    f[rng.integers(0, f.size, 3)] = [np.inf, -np.inf, np.nan]
    a, b = (_run(wl, f, tmem, precision, 0, active, (1,)) for tmem in (1, 0))
    assert np.array_equal(a, b, equal_nan=True)
