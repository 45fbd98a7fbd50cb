"""Lane groups: evaluators that give a flight to several lanes (EvalGroup3D: a warp per
flight below 10 000 flights, eight lanes above).  The flight bars of test_gpu_parity
against the oracle, at batch sizes around the groups, the blocks and the change of
group size, with impulse counts that leave lanes without an impulse, and with 9 per
cell, which takes the evaluator without groups."""
import numpy as np
import pytest

from gpis_extend_gb300 import abi, runtime, workloads
from oracle import oracle
from test_gpu_parity import flights_vs_oracle

pytestmark = pytest.mark.gpu


def medium_3d(impulses, **kw):
    return workloads.sphere_medium(one_d=False, impulse_density=float(impulses), **kw)


@pytest.mark.parametrize("n,impulses,kw", [
    (1, 8, {}), (7, 1, {}), (33, 8, dict(context=abi.CTX_RENEWAL)), (257, 5, dict(impulse_xyz_order=1)),
    (9999, 8, dict(context=abi.CTX_RENEWAL)), (10000, 8, {}), (12289, 3, dict(aniso=(1.0, 0.6, 1.4))), (300, 9, {})])
def test_gpu_3d_groups_match_oracle(n, impulses, kw):
    desc = medium_3d(impulses, **kw)
    prim = workloads.sphere_flights(n, desc)
    with runtime.Context(desc) as ctx:
        rec = ctx.trace_host(prim)
        flights_vs_oracle(desc, prim, rec)
        sec, _ = workloads.secondary_flights(prim, oracle.trace_flights(desc, prim), desc)
        if sec.n:
            flights_vs_oracle(desc, sec, ctx.trace_host(sec))


def test_gpu_3d_group_sizes_agree():
    """Both group sizes on the same flights: decisions and hits are taken on the precise
    values, so they agree bit for bit; a miss value is a sum in another order (24 terms of
    magnitude below 1 within about 1e-6 of each other after the normalisation)."""
    desc = medium_3d(8, context=abi.CTX_RENEWAL)
    prim = workloads.sphere_flights(10500, desc)
    idx = np.arange(0, prim.n, 3)
    with runtime.Context(desc) as ctx:
        many = ctx.trace_host(prim)[idx]
        few = ctx.trace_host(prim.subset(idx))
    a, b = abi.unpack_results(many), abi.unpack_results(few)
    for name in ("status", "steps", "hit", "t", "gp_id"):
        assert np.array_equal(a[name], b[name]), name
    hit = a["hit"]
    assert np.array_equal(many[hit].view(np.uint32), few[hit].view(np.uint32))
    assert np.abs(a["value"] - b["value"]).max() <= 2e-6
