"""Whole runs of steps in one launch with several tiles per warp, alone and for
a batch's members side by side, against a launch per stage (the tensor memory
off).  The same operations on every line in the same order: the tolerance is
zero bits, NaNs included.
"""
import numpy as np
import pytest

from bfvm import Batch, Microenvironment
from bfvm import workloads as W

pytestmark = pytest.mark.gpu


def _solve(wl, tmem, precision, chain=0, active=None, field=None):
    me = Microenvironment.from_workload(wl, precision=precision, upload=False)
    if active is not None:
        me.set_dirichlet_activation(active)
    me.upload_field(wl.field0 if field is None else field)
    me.set_fp64_chain(chain)
    me.set_sweep_tmem(tmem)
    return me


def _run(wl, tmem, precision, chain, active, field=None):
    me = _solve(wl, tmem, precision, chain, active, field)
    for n in (4, 5):
        me.simulate_diffusion_decay(n, sources=True)
    out = me.download_field()
    me.close()
    return out


# More than eight tiles per SM (the fewest that do so among them), lines about
# the batches of 16 values, x rows of one and of several 128-byte lines, last
# tiles of one line, face rows only (nz of 2), the longest lines that leave
# three warps an SM and longer ones, warps half busy and less, more than 32
# agents to a tile, more agents than this form takes.
SHAPES = [(64, 64, 75, 8, 900), (33, 97, 95, 5, 20000), (97, 33, 81, 6, 3000), (100, 113, 64, 6, 300),
          (255, 60, 62, 3, 5000), (40, 36, 300, 4, 700), (310, 41, 33, 5, 700), (400, 1200, 2, 1, 4000),
          (129, 127, 128, 3, 40000)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision,chain", [("fp64", 0), ("fp64", 1), ("fp32", 0), ("fp32", 1)])
def test_several_tiles_per_warp_equal_a_launch_per_stage(shape, precision, chain):
    nx, ny, nz, S, agents = shape
    wl = W.small_random(500 + nx + ny + nz, nx=nx, ny=ny, nz=nz, S=S, n_agents=agents, steps=3)
    for active in (np.ones(S, np.uint8), np.arange(S, dtype=np.uint8) % 2):
        a, b = (_run(wl, tmem, precision, chain, active) for tmem in (1, 0))
        assert np.array_equal(a, b), (shape, precision, chain, active)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_several_tiles_per_warp_special_values(precision):
    wl = W.small_random(8, nx=66, ny=65, nz=75, S=8, n_agents=200, steps=2)
    active = np.arange(8, dtype=np.uint8) % 2
    rng = np.random.default_rng(5)
    f = wl.field0.copy()
    odd = [-1.0, 0.0, -0.0, 5e-324, 2.0 ** -960, 2.0 ** -961, -2.0 ** -970, 1e30]
    f[rng.integers(0, f.size, f.size // 50)] = rng.choice(odd, f.size // 50)
    f[rng.integers(0, f.size, 3)] = [np.inf, -np.inf, np.nan]
    a, b = (_run(wl, tmem, precision, 0, active, f) for tmem in (1, 0))
    assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("members", [1, 3, 53])
def test_batch_members_side_by_side_equal_solves_alone(precision, members):
    """Members of one tile and of many, more of them than one launch takes, one
    that keeps to the other forms (agents tracked), runs of one step, of less
    and of more than the batch's graph, and of more than one launch takes."""
    rng = np.random.default_rng(members)
    wls = [W.small_random(40 + q, nx=int(rng.integers(1, 60)), ny=int(rng.integers(1, 60)), nz=int(rng.integers(2, 60)),
                          S=int(rng.integers(1, 7)), n_agents=int(rng.integers(1, 600)), steps=1)
           for q in range(members)]
    for tracked in (False, True):
        batch, mes = Batch(precision), []
        batch.set_schedule(mode=2, graph_steps=4)
        batch.set_direct_threshold(50000)
        for q, wl in enumerate(wls):
            me = _solve(wl, 1, precision)
            if tracked and q == members - 1:
                me.set_track_internalized_substrates(True)
            batch.add(me)
            mes.append(me)
        steps = (1, 3, 6) if members > 3 else (1, 6, 67)
        for n in steps:
            batch.step(n, sources=True)
        batch.synchronize()
        for wl, me in zip(wls, mes):
            solo = _solve(wl, 0, precision)
            solo.simulate_diffusion_decay(sum(steps), sources=True)
            assert np.array_equal(me.download_field(), solo.download_field()), (wl.field0.size, tracked)
            solo.close()
        batch.close()
        for me in mes:
            me.close()
