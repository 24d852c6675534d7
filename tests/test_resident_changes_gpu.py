"""What may change between runs of steps that go in one launch, also where that
launch has been captured into a graph: the results follow, bit for bit, those
of a solve that takes a launch per stage (the tensor memory off)."""
import numpy as np
import pytest
import torch

from bfvm import Batch, Microenvironment
from bfvm import workloads as W

pytestmark = pytest.mark.gpu


def _solve(wl, precision, tmem=1):
    me = Microenvironment.from_workload(wl, precision=precision)
    me.set_sweep_tmem(tmem)
    return me


def _small(q, S=3):
    return W.small_random(880 + q, nx=30 + 3 * q, ny=25 + q, nz=20 + 2 * q, S=S, n_agents=100, steps=1)


# From none to all, and from all to one: more face lines, and fewer.
ACTIVATIONS = [np.zeros(3, np.uint8), np.ones(3, np.uint8), np.array([0, 0, 1], np.uint8)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_captured_batch_follows_the_activation(precision):
    """A batch with members in the one launch and one beside it (its agents
    tracked), so that its steps replay a graph: an activation that changes
    between two calls takes effect in the replay."""
    wls = [_small(q) for q in range(4)]
    batch = Batch(precision)
    batch.set_schedule(mode=2, graph_steps=4)
    mes, solos = [], []
    for q, wl in enumerate(wls):
        for tmem, to in ((1, mes), (0, solos)):
            me = _solve(wl, precision, tmem)
            me.set_dirichlet_activation(ACTIVATIONS[0])
            me.set_track_internalized_substrates(q == 3)
            to.append(me)
        batch.add(mes[-1])
    for active in ACTIVATIONS + ACTIVATIONS[:1]:
        for me in mes + solos:
            me.set_dirichlet_activation(active)
        batch.step(8, sources=True)
        batch.synchronize()
        for q, (me, solo) in enumerate(zip(mes, solos)):
            solo.simulate_diffusion_decay(8, sources=True)
            assert np.array_equal(me.download_field(), solo.download_field()), (q, active)
    batch.close()
    for me in mes + solos:
        me.close()


@pytest.mark.parametrize("shape", [(40, 36, 30), (100, 100, 96)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_captured_run_follows_the_activation(shape, precision):
    """The caller's own capture of a run in one launch, one tile per warp and
    several."""
    nx, ny, nz = shape
    wl = W.small_random(nx, nx=nx, ny=ny, nz=nz, S=3, n_agents=300, steps=1)
    me, solo = _solve(wl, precision), _solve(wl, precision, 0)
    stream = torch.cuda.Stream()
    me.set_stream(stream.cuda_stream)
    me.simulate_diffusion_decay(5, sources=True)
    me.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        me.simulate_diffusion_decay(5, sources=True)
    solo.simulate_diffusion_decay(5, sources=True)
    for active in ACTIVATIONS:
        for m in (me, solo):
            m.set_dirichlet_activation(active)
        with torch.cuda.stream(stream):
            graph.replay()
        me.synchronize()
        solo.simulate_diffusion_decay(5, sources=True)
        assert np.array_equal(me.download_field(), solo.download_field()), active
    del graph
    me.close()
    solo.close()


SETTINGS = {
    "timing": lambda me, on: me.timing_enable(not on),
    "tmem": lambda me, on: me.set_sweep_tmem(1 if on else 0),
    "schedule": lambda me, on: me.set_sweep_schedule(1 if on else 2),
    "streams": lambda me, on: me.set_substrate_streams(1 if on else 2),
    "launch": lambda me, on: me.set_launch(32 if on else 64, 32, 32),
    "fused": lambda me, on: me.set_fused_sources(not on),
    "chain": lambda me, on: me.set_fp64_chain(0 if on else 1),
}


@pytest.mark.parametrize("setting", sorted(SETTINGS))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_follows_its_members_settings(setting, precision):
    """A member's launch setting changes between the steps of a batch and goes
    back: the member leaves the one launch or returns to it, and every member
    goes on step by step, in calls that replay the graph and in ones that do
    not.  50 members: the one launch is two."""
    wls = [W.small_random(990 + q, nx=9 + q % 7, ny=8 + q % 5, nz=7 + q % 3, S=2, n_agents=20, steps=1)
           for q in range(50)]
    batch = Batch(precision)
    batch.set_schedule(mode=2, graph_steps=4)
    mes, solos = ([_solve(wl, precision, tmem) for wl in wls] for tmem in (1, 0))
    for me in mes:
        batch.add(me)
    for on in (True, False, True):
        SETTINGS[setting](mes[-1], on)
        if setting == "chain":
            SETTINGS[setting](solos[-1], on)
        for n in (2, 4):
            batch.step(n, sources=True)
        batch.synchronize()
        for q, (me, solo) in enumerate(zip(mes, solos)):
            solo.simulate_diffusion_decay(6, sources=True)
            assert np.array_equal(me.download_field(), solo.download_field()), (q, on)
    batch.close()
    for me in mes + solos:
        me.close()
