"""Which lines chain 2 solves by the partition method is the solve's own: neither
the launch settings nor how its steps are shared out over calls change a bit,
and a threshold that was set holds on every grid."""
import numpy as np
import pytest

from bfvm import Microenvironment
from bfvm import workloads as W

pytestmark = pytest.mark.gpu

STEPS = 8


def _run(wl, precision, change=None, calls=(STEPS,), chain=2, min_line=None):
    me = Microenvironment.from_workload(wl, precision=precision)
    me.set_fp64_chain(chain)
    if min_line is not None:
        me.set_partition_min_line(min_line)
    if change is not None:
        change(me)
    for n in calls:
        me.simulate_diffusion_decay(n, sources=True)
    out = me.download_field()
    me.close()
    return out


CHANGES = {
    "single steps": (None, (1,) * STEPS),
    "no tensor memory": (lambda me: me.set_sweep_tmem(0), (STEPS,)),
    "a launch per tile": (lambda me: me.set_sweep_schedule(0), (STEPS,)),
    "persistent sweeps": (lambda me: me.set_sweep_schedule(2), (STEPS,)),
    "two streams": (lambda me: me.set_substrate_streams(2), (STEPS,)),
    "timing": (lambda me: me.timing_enable(True), (STEPS,)),
    "tiles": (lambda me: me.set_launch(16, 32, 16), (STEPS,)),
}


# Lines past the default threshold: on a grid that one launch could take, of few
# tiles and of many, so many that half the substrates have few, and lines that
# are always partitioned.
@pytest.mark.parametrize("shape,precision", [((64, 480, 32, 4), "fp32"), ((40, 33, 500, 2), "fp32"),
                                             ((64, 520, 100, 2), "fp64"), ((33, 520, 40, 1), "fp64"),
                                             ((36, 40, 600, 2), "fp64")])
def test_launch_settings_keep_the_bits(shape, precision):
    nx, ny, nz, S = shape
    wl = W.small_random(ny, nx=nx, ny=ny, nz=nz, S=S, n_agents=300, steps=1)
    expect = _run(wl, precision)
    for name, (change, calls) in CHANGES.items():
        assert np.array_equal(_run(wl, precision, change, calls), expect), name


@pytest.mark.parametrize("shape", [(40, 36, 30, 2), (64, 64, 80, 8), (9, 70, 5, 1)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_a_set_threshold_holds_on_small_grids(shape, precision):
    """The partitioned sweeps' bits, however the steps are called, and not those
    of the serial chain, which a threshold past the lines gives."""
    nx, ny, nz, S = shape
    wl = W.small_random(17, nx=nx, ny=ny, nz=nz, S=S, n_agents=100, steps=1)
    for change, calls in CHANGES.values():
        assert np.array_equal(_run(wl, precision, change, calls, min_line=1), _run(wl, precision, min_line=1))
    serial = _run(wl, precision, min_line=max(ny, nz) + 1)
    assert np.array_equal(serial, _run(wl, precision, chain=1))
    assert not np.array_equal(serial, _run(wl, precision, min_line=1))
