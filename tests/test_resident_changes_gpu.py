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
