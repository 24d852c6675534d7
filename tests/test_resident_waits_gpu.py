"""The grid-wide barrier of runs in one launch: a wait that runs out ends the run
with a status and leaves the solve usable.  And planes of one row or column,
whose sweeps have lines of one value."""
import numpy as np
import pytest

from bfvm import Batch, Microenvironment, kernel_launches
from bfvm import workloads as W
from bfvm._lib import BFVM_ERR_TIMEOUT, BFVM_OK

pytestmark = pytest.mark.gpu

LIMIT_TEST_NS = 1000
LIMIT_DEFAULT_NS = 2_000_000_000

# As many agents in one voxel as still go tile by tile: one warp takes tens of
# microseconds over them, and the other CTAs wait.
STACK = 190


def _workload(nx, ny, nz, S):
    return W.small_random(nx + 2 * ny, nx=nx, ny=ny, nz=nz, S=S, n_agents=0, steps=1)


def _solve(wl, precision, tmem=1):
    me = Microenvironment.from_workload(wl, precision=precision)
    me.set_sweep_tmem(tmem)
    nx, ny, nz, S = me.shape
    rng = np.random.default_rng(nx)
    me.set_agents_from_rates(voxel=np.full(STACK, (nx // 2 * ny + ny // 2) * nz + nz // 2, np.int32),
                             volume=np.full(STACK, 2494.0), secretion=rng.random((STACK, S)),
                             uptake=rng.random((STACK, S)), saturation=np.ones((STACK, S)),
                             net_export=np.zeros((STACK, S)))
    return me


def _step(me, n):
    (me.simulate_diffusion_decay_2d if me.shape[2] == 1 else me.simulate_diffusion_decay)(n, sources=True)


def _expect(wl, precision, n):
    solo = _solve(wl, precision, 0)
    _step(solo, n)
    out = solo.download_field()
    solo.close()
    return out


# One tile per warp, several, and a plane.
@pytest.mark.parametrize("shape", [(50, 50, 50, 2), (128, 128, 128, 3), (90, 127, 1, 2)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_barrier_that_gives_up_leaves_the_solve_usable(shape, precision):
    """With a limit of 1 us the CTAs that wait for the stack's give up, in both
    launches of a call of 70 steps; the status is reported once, and from its
    initial field the solve steps bit for bit again."""
    wl = _workload(*shape)
    me = _solve(wl, precision)
    _step(me, 5)
    me.synchronize()
    before = kernel_launches()
    assert me.L.bfvm_set_wait_limit_ns(0, LIMIT_TEST_NS) == BFVM_OK
    try:
        _step(me, 70)
        assert kernel_launches() - before == 2
        assert me.L.bfvm_synchronize(me.h) == BFVM_ERR_TIMEOUT
    finally:
        assert me.L.bfvm_set_wait_limit_ns(0, LIMIT_DEFAULT_NS) == BFVM_OK
    assert me.L.bfvm_synchronize(me.h) == BFVM_OK
    me.upload_field(wl.field0)
    _step(me, 70)
    assert np.array_equal(me.download_field(), _expect(wl, precision, 70))
    me.close()


def test_a_batch_recovers_from_a_barrier_that_gives_up():
    wls = [_workload(30 + q, 40, 33, 2) for q in range(3)]
    mes = [_solve(wl, "fp32") for wl in wls]
    batch = Batch("fp32")
    batch.set_schedule(mode=2)
    for me in mes:
        batch.add(me)
    batch.step(2, sources=True)
    batch.synchronize()
    assert batch.L.bfvm_set_wait_limit_ns(0, LIMIT_TEST_NS) == BFVM_OK
    try:
        batch.step(6, sources=True)
        assert batch.L.bfvm_batch_synchronize(batch.h) == BFVM_ERR_TIMEOUT
    finally:
        assert batch.L.bfvm_set_wait_limit_ns(0, LIMIT_DEFAULT_NS) == BFVM_OK
    assert batch.L.bfvm_batch_synchronize(batch.h) == BFVM_OK
    for wl, me in zip(wls, mes):
        me.upload_field(wl.field0)
    batch.step(6, sources=True)
    batch.synchronize()
    for wl, me in zip(wls, mes):
        assert np.array_equal(me.download_field(), _expect(wl, "fp32", 6))
    batch.close()
    for me in mes:
        me.close()


@pytest.mark.parametrize("shape", [(60, 1, 1, 2), (1, 60, 1, 2), (1, 1, 1, 1), (130, 1, 1, 3)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_planes_of_one_row_or_column(shape, precision):
    nx, ny, nz, S = shape
    wl = W.small_random(nx + 2 * ny, nx=nx, ny=ny, nz=nz, S=S, n_agents=40, steps=1)
    nodes = (np.array([0, nx * ny - 1], np.int32)[: nx * ny], np.full((2, S), 7.0)[: nx * ny],
             np.ones((2, S), np.uint8)[: nx * ny])
    for nd in (None, nodes):
        out = []
        for tmem in (1, 0):
            me = Microenvironment.from_workload(wl, precision=precision)
            me.set_sweep_tmem(tmem)
            if nd is not None:
                me.set_dirichlet_nodes(*nd)
            for n in (1, 3):
                me.simulate_diffusion_decay_2d(n, sources=True)
            out.append(me.download_field())
            me.close()
        assert np.array_equal(*out), nd is None
