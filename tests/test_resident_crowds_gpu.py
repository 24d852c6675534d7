"""Agents that crowd into few tiles of a run in one launch go ahead of the x sweep,
by all threads, instead of tile by tile: the same bits as a launch per stage
(the tensor memory off)."""
import numpy as np
import pytest

from bfvm import Batch, Microenvironment
from bfvm import workloads as W

pytestmark = pytest.mark.gpu


def _solve(wl, voxel, precision, tmem):
    rng = np.random.default_rng(voxel.size)
    n, S = voxel.size, wl.S
    me = Microenvironment.from_workload(wl, precision=precision)
    me.set_sweep_tmem(tmem)
    me.set_agents_from_rates(voxel=voxel, volume=np.full(n, 2494.0), secretion=rng.random((n, S)),
                             uptake=10 * rng.random((n, S)), saturation=np.ones((n, S)), net_export=rng.random((n, S)))
    return me


def _crowd(shape, n, seed):
    """n agents in the rows of one x tile, a third of them in one voxel of it."""
    nx, ny, nz, _ = shape
    rng = np.random.default_rng(seed)
    row = (ny * nz // 2) // 32 * 32 + rng.integers(0, min(32, ny * nz), n)
    row[: n // 3] = row[0]
    i = rng.integers(0, nx, n)
    i[: n // 3] = nx // 2
    return ((i * ny + row % ny) * nz + row // ny).astype(np.int32)


# One tile per warp, several, and a plane; as many agents as a tile still takes
# and one more, and many of them.
SHAPES = [(40, 36, 30, 2), (64, 64, 110, 8), (90, 127, 1, 2)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("agents", [192, 193, 3000])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_crowds_equal_a_launch_per_stage(shape, agents, precision):
    nx, ny, nz, S = shape
    wl = W.small_random(nx + agents, nx=nx, ny=ny, nz=nz, S=S, n_agents=0, steps=1)
    out = []
    for tmem in (1, 0):
        me = _solve(wl, _crowd(shape, agents, 3), precision, tmem)
        for n in (1, 4):
            if nz == 1:
                me.simulate_diffusion_decay_2d(n, sources=True)
            else:
                me.simulate_diffusion_decay(n, sources=True)
        out.append(me.download_field())
        me.close()
    assert np.array_equal(*out)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_crowds_in_a_batch_equal_solves_alone(precision):
    """A crowded member beside ones that are not; the list changes between two
    calls, to one that is not crowded either."""
    shapes = [(40, 36, 30, 2), (64, 64, 80, 8), (33, 30, 20, 1)]
    wls = [W.small_random(60 + q, nx=s[0], ny=s[1], nz=s[2], S=s[3], n_agents=0, steps=1)
           for q, s in enumerate(shapes)]
    voxels = [_crowd(shapes[0], 800, 1), _crowd(shapes[1], 190, 2), _crowd(shapes[2], 193, 3)]
    mes, solos = ([_solve(wl, v, precision, tmem) for wl, v in zip(wls, voxels)] for tmem in (1, 0))
    batch = Batch(precision)
    batch.set_schedule(mode=2)
    for me in mes:
        batch.add(me)
    for again in (False, True):
        if again:
            for group in (mes, solos):
                group[0].set_agents_from_rates(voxel=voxels[0][:50], volume=np.full(50, 2494.0),
                                               secretion=np.ones((50, 2)), uptake=np.ones((50, 2)),
                                               saturation=np.ones((50, 2)), net_export=np.zeros((50, 2)))
        batch.step(5, sources=True)
        batch.synchronize()
        for me, solo in zip(mes, solos):
            solo.simulate_diffusion_decay(5, sources=True)
            assert np.array_equal(me.download_field(), solo.download_field()), again
    batch.close()
    for me in mes + solos:
        me.close()
