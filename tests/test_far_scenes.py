"""Step skipping away from the origin: a step's point is rounded to float, at 10^4 units by
5e-4, far more than the noise of a smooth surface changes over a step, and the second-order
reach of plain media has to allow for it.  The steps taken are the oracle's on 99.95 % of the
flights, as in scenes around the origin (its evaluation rounds the points in the same way)."""
import numpy as np
import pytest

from gpis_extend_gb300 import abi, workloads
from oracle import oracle

pytestmark = pytest.mark.gpu

FAR = np.array([10000.0, 0.0, -8000.0])


@pytest.mark.parametrize("n", [8000, 40_000])
@pytest.mark.parametrize("sigma", [0.05, 5e-4, 5e-5])
@pytest.mark.parametrize("mean", ["sphere", "torus"])
def test_gpu_far_scene_steps(mean, sigma, n):
    """Eight lanes and one lane a flight."""
    from gpis_extend_gb300 import runtime
    params = tuple(FAR) + ((1.0,) if mean == "sphere" else (1.0, 0.35))
    desc = workloads.sphere_medium(sigma=sigma, mean_params=params,
                                   mean_kind=abi.MEAN_SPHERE if mean == "sphere" else abi.MEAN_TORUS)
    prim = workloads.sphere_flights(n, desc)
    prim.origin_near[:, :3] = (prim.origin_near[:, :3].astype(np.float64) + FAR).astype(np.float32)
    with runtime.Context(desc) as ctx:
        ctx.counters(reset=True)
        g = abi.unpack_results(ctx.trace_host(prim))
        cnt = ctx.counters(reset=True)
    c = abi.unpack_results(oracle.trace_flights(desc, prim))
    differ = np.mean(g["steps"] != c["steps"])
    print(mean, sigma, n, "steps differ", differ, "skipped", cnt["skipped_steps"] / cnt["steps"])
    assert np.mean(g["hit"] == c["hit"]) >= 0.9999
    assert differ <= 5e-4
    assert cnt["skipped_steps"] > 0.5 * cnt["steps"]
