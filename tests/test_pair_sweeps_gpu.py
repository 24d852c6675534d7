"""The sweeps that run two tiles per warp against the general path.

Schedule 2 launches them whatever the tile count; with the tensor memory off
the shared-memory and per-tile sweeps run instead.  Both do the same operations
on every line in the same order, so the tolerance is zero bits, NaNs included.
"""
import numpy as np
import pytest

from bfvm import Microenvironment
from bfvm import workloads as W

pytestmark = pytest.mark.gpu


def _run(wl, field, tmem, precision, chain, active):
    me = Microenvironment.from_workload(wl, precision=precision, upload=False)
    me.set_dirichlet_activation(active)
    me.upload_field(field)
    me.set_fp64_chain(chain)
    me.set_sweep_schedule(2)
    me.set_sweep_tmem(tmem)
    me.simulate_diffusion_decay(wl.steps)
    out = me.download_field()
    me.close()
    return out


# Line lengths about the changes of form: whole and ragged last chunks of 16
# (FP64) and 32 (FP32) values, 8 | 9 and 16 | 17 chunks, lines past tensor
# memory; x tiles with two, many and only face rows (ny < 32, nz of 1 and 2);
# packed tiles of every width; more tiles than one round of the rings.
SHAPES = [(64, 49, 50, 2), (128, 33, 129, 1), (129, 128, 40, 2), (176, 161, 34, 1), (177, 31, 33, 2), (256, 35, 256, 1),
          (257, 20, 2, 3), (272, 65, 1, 2), (36, 272, 257, 1), (48, 500, 33, 1), (224, 224, 70, 3), (34, 33, 900, 1),
          (1000, 36, 5, 1), (97, 211, 143, 2), (1, 300, 33, 2), (33, 1, 300, 2)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision,chain", [("fp64", 0), ("fp64", 1), ("fp32", 0), ("fp32", 1)])
def test_pair_sweeps_equal_the_general_path(shape, precision, chain):
    nx, ny, nz, S = shape
    wl = W.small_random(7000 + nx + ny + nz, nx=nx, ny=ny, nz=nz, S=S, n_agents=0, steps=2)
    for active in (np.ones(S, np.uint8), np.arange(S, dtype=np.uint8) % 2):
        a, b = (_run(wl, wl.field0, tmem, precision, chain, active) for tmem in (1, 0))
        assert np.array_equal(a, b), (shape, precision, chain, active)


@pytest.mark.parametrize("shape", [(200, 64, 33, 2), (36, 300, 64, 1), (128, 70, 200, 1)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_pair_sweeps_special_values(shape, precision):
    """Inputs that the exactness screen sends back (negative, zero, -0,
    subnormal and about 2^-960), infinities and NaNs: a tile redone or not,
    the same bits."""
    nx, ny, nz, S = shape
    wl = W.small_random(31, nx=nx, ny=ny, nz=nz, S=S, n_agents=0, steps=2)
    rng = np.random.default_rng(5)
    f = wl.field0.copy()
    odd = [-1.0, 0.0, -0.0, 5e-324, 2.0 ** -960, 2.0 ** -961, -2.0 ** -970, 1e30]
    f[rng.integers(0, f.size, f.size // 50)] = rng.choice(odd, f.size // 50)
    active = np.arange(S, dtype=np.uint8) % 2
    a, b = (_run(wl, f, tmem, precision, 0, active) for tmem in (1, 0))
    assert np.array_equal(a, b)
    f[rng.integers(0, f.size, 5)] = [np.inf, -np.inf, np.nan, np.inf, np.nan]
    a, b = (_run(wl, f, tmem, precision, 0, active) for tmem in (1, 0))
    assert np.array_equal(a, b, equal_nan=True)
