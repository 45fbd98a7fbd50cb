"""The level weights of the multi-resolution grid: (1 - f) / d and f / d with d = sqrt(1 - 2 f
+ 2 f f), taken in double and rounded to float as the reference does, in the fast passes
too.  With a constant length scale the medium is the two-octave medium whose octaves are
the two levels, with the weights as amplitudes; a power of two as sigma scales exactly, so
the records of misses, whose value is the fast evaluator's, are equal bit for bit."""
import numpy as np
import pytest

from gpis_extend_gb300 import abi, workloads
from oracle import oracle

pytestmark = pytest.mark.gpu

SIGMA = 2.0 ** -5


def two_octaves(desc):
    info, seeds = oracle.level_ratio(desc, np.zeros(3, np.float32))
    # the weights from the levels in double, rounded once
    s0, s1 = np.float32(info[0]), np.float32(info[1])
    f = float((np.float32(desc.ls_params[0]) - s0) / (s1 - s0))
    den = np.sqrt(1.0 - 2.0 * f + 2.0 * f * f)
    w = [np.float32((1.0 - f) / den), np.float32(f / den)]
    return workloads.torus_plane_medium(nonstationary=False, length_scale=1.0, sigma=SIGMA, n_octaves=2,
                                        octave_sigma=[float(SIGMA * v) for v in w], octave_scale=[float(s0), float(s1)],
                                        octave_seed=[int(s) for s in seeds])


@pytest.mark.parametrize("n", [3000, 14_000, 24_000])
@pytest.mark.parametrize("ls", [0.041, 0.057, 0.0733, 0.09, 0.1127, 0.1361, 0.149, 0.1571])
def test_gpu_level_weights_round_once(n, ls):
    """A warp, eight lanes and one lane per flight."""
    from gpis_extend_gb300 import runtime
    desc = workloads.torus_plane_medium(octaves=1, multires=1, sigma=SIGMA, ls_params=(ls, 0.0, 1.0, 1.0))
    octaves = two_octaves(desc)
    prim = workloads.torus_flights(n, desc)
    with runtime.Context(desc) as ctx:
        levels = abi.unpack_results(ctx.trace_host(prim))
    with runtime.Context(octaves) as ctx:
        octs = abi.unpack_results(ctx.trace_host(prim))
    miss = ~octs["hit"]
    assert miss.sum() > n // 40
    # (the gradient at the end point draws its random part per octave)
    for name in ("hit", "steps", "status"):
        assert np.array_equal(levels[name], octs[name]), name
    for name in ("t", "value"):
        assert np.array_equal(levels[name].view(np.uint32), octs[name].view(np.uint32)), name
