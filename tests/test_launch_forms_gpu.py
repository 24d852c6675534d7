"""Which form a run of steps takes, by the launches it makes (bfvm_kernel_launches)
and by the kernels that the GPU ran, and that the forms give the same bits."""
import numpy as np
import pytest
import torch

from bfvm import Batch, Microenvironment, kernel_launches
from bfvm import workloads as W

pytestmark = pytest.mark.gpu


def _launches(call):
    before = kernel_launches()
    call()
    return kernel_launches() - before


def _kernels(call):
    """The kernels' names, in the order of their launches."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "kernel" in e.name]


def _small(q=0, S=2):
    return W.small_random(4400 + q, nx=40 + q, ny=36, nz=30, S=S, n_agents=300, steps=1)


# The sizes and the steps of a call, its launches, and the kernel: one tile per
# warp, several, more steps than one launch takes, a plane, and past the L2.
@pytest.mark.parametrize("shape,steps,launches,kernel", [
    ((40, 36, 30, 2), 10, 1, "resident_kernel"), ((40, 36, 30, 2), 131, 3, "resident_kernel"),
    ((100, 100, 96, 3), 10, 1, "resident_many_kernel"), ((90, 127, 1, 3), 10, 1, "resident_kernel"),
    ((256, 200, 300, 4), 1, 4, "sweep_pair_kernel")])
def test_forms_of_a_run(shape, steps, launches, kernel):
    nx, ny, nz, S = shape
    wl = W.small_random(nx, nx=nx, ny=ny, nz=nz, S=S, n_agents=200, steps=1)
    me = Microenvironment.from_workload(wl, precision="fp32" if nx == 100 else "fp64")
    step = me.simulate_diffusion_decay_2d if nz == 1 else me.simulate_diffusion_decay
    step(1, sources=True)
    assert _launches(lambda: step(steps, sources=True)) == launches
    names = _kernels(lambda: step(steps, sources=True))
    if not names:
        pytest.skip("the profiler records no kernels here")
    assert len(names) == launches and any(kernel in n for n in names), names
    me.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_graphs_follow_agents_and_schedules(precision):
    """A solve that asks for a launch per stage replays its captured steps, and
    captures them again after a new agent list and a new schedule."""
    wl = _small(1)
    me, solo = (Microenvironment.from_workload(wl, precision=precision) for _ in range(2))
    me.set_fused_sources(False)
    rng = np.random.default_rng(3)
    n = wl.n_agents // 2
    rates = dict(voxel=wl.agent_voxel[:n], volume=np.full(n, 2494.0), secretion=rng.random((n, 2)),
                 uptake=rng.random((n, 2)), saturation=np.ones((n, 2)), net_export=rng.random((n, 2)))
    for change in (lambda m: None, lambda m: m.set_agents_from_rates(**rates), lambda m: m.set_sweep_schedule(2)):
        change(me)
        change(solo)
        me.synchronize()
        assert _launches(lambda: me.simulate_diffusion_decay(40, sources=True)) == 40 * 4
        for _ in range(40):
            solo.simulate_diffusion_decay(1, sources=True)
        assert np.array_equal(me.download_field(), solo.download_field())
    me.close()
    solo.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_members_side_by_side_are_one_launch(precision):
    """Small members in one launch, more of them than one launch takes, and one
    that is tracked beside them through the batched sweeps, called step by step
    and replayed; with a threshold set, all in the batched sweeps or direct."""
    wls = [W.small_random(4500 + q, nx=9 + q % 40, ny=20, nz=12, S=2, n_agents=20, steps=1) for q in range(53)]
    for tracked in (False, True):
        mes = [Microenvironment.from_workload(wl, precision=precision) for wl in wls]
        mes[-1].set_track_internalized_substrates(tracked)
        batch = Batch(precision)
        batch.set_schedule(mode=2, graph_steps=4)
        for me in mes:
            batch.add(me)
        batch.step(1, sources=True)
        beside = 3 if tracked else 0
        assert _launches(lambda: batch.step(1, sources=True)) == 2 + beside
        # not tracked: nothing to replay; else three steps, then the graph of four
        assert _launches(lambda: batch.step(7, sources=True)) == (4 + 7 * beside if tracked else 2)
        batch.set_direct_threshold(1 << 20)
        batch.step(1, sources=True)
        assert _launches(lambda: batch.step(5, sources=True)) == 5 * 3
        batch.set_direct_threshold(1)
        batch.step(1, sources=True)
        assert _launches(lambda: batch.step(5, sources=True)) == 5 * 4 * len(mes)
        batch.synchronize()
        for q in (0, 30, 52):
            solo = Microenvironment.from_workload(wls[q], precision=precision)
            solo.set_fused_sources(False)
            solo.simulate_diffusion_decay(21, sources=True)
            assert np.array_equal(mes[q].download_field(), solo.download_field()), q
            solo.close()
        batch.close()
        for me in mes:
            me.close()


# Runs that fill the SMs: a tile per warp and several, with enough to do; and those
# that other streams' solves would wait for: few warps, short lines, idle lanes,
# few values, FP64 in calls that replay a graph, dense agents, a call of 3 steps;
# and planes.
@pytest.mark.parametrize("shape,agents,steps,one", [
    ((50, 50, 50, 8), 300, 10, True), ((50, 50, 50, 8), 300, 20, "fp32"), ((50, 50, 50, 8), 300, 3, False),
    ((50, 50, 50, 8), 9000, 10, False), ((128, 100, 100, 2), 300, 10, True), ((60, 60, 60, 6), 300, 10, False),
    ((32, 32, 32, 24), 300, 10, False), ((128, 64, 64, 4), 300, 10, "fp32"), ((64, 64, 64, 16), 300, 10, "fp64"),
    ((128, 128, 128, 2), 300, 20, True), ((129, 127, 128, 3), 300, 20, True), ((40, 36, 300, 4), 300, 10, False),
    ((600, 400, 1, 4), 300, 10, "fp32"), ((100, 130, 1, 4), 300, 10, True)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_runs_that_fill_the_gpu(shape, agents, steps, one, precision):
    nx, ny, nz, S = shape
    wl = W.small_random(steps + nx, nx=nx, ny=ny, nz=nz, S=S, n_agents=agents, steps=1)
    me, solo = (Microenvironment.from_workload(wl, precision=precision) for _ in range(2))
    solo.set_sweep_tmem(0)
    step = "simulate_diffusion_decay" + ("_2d" if nz == 1 else "")
    launches = _launches(lambda: getattr(me, step)(steps, sources=True))
    assert launches == (1 if one in (True, precision) else (3 if nz == 1 else 4) * steps)
    getattr(solo, step)(steps, sources=True)
    assert np.array_equal(me.download_field(), solo.download_field())
    me.close()
    solo.close()
