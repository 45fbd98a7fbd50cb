"""Lane groups: evaluators that give a flight to several lanes (EvalGroup3D: a warp per
flight below 10 000 flights, eight lanes above; EvalGroup1D: eight lanes in the resume
passes of 1D media while their queues are short).  The flight bars of test_gpu_parity
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


MEDIA_1D = {
    "sphere": (workloads.sphere_medium, workloads.sphere_flights, 1.5),
    "one_impulse": (lambda: workloads.sphere_medium(impulse_density=1.0), workloads.sphere_flights, 1.5),
    "octaves": (workloads.torus_plane_medium, workloads.torus_flights, 2.0),
    "multires": (lambda: workloads.torus_plane_medium(octaves=1, multires=1), workloads.torus_flights, 2.0),
    "nonstationary": (lambda: workloads.torus_plane_medium(octaves=1), workloads.torus_flights, 2.0),
    "xy": (lambda: workloads.sphere_medium(correlation_xy=1, aniso=(1.0, 0.7, 1.3)), workloads.sphere_flights, 1.5),
    "nine_impulses": (lambda: workloads.sphere_medium(impulse_density=9.0), workloads.sphere_flights, 1.5),
}


@pytest.mark.parametrize("kind,n", [("sphere", 1), ("sphere", 31), ("sphere", 65537), ("one_impulse", 1000),
                                    ("octaves", 2049), ("multires", 1025), ("nonstationary", 3001), ("xy", 5000),
                                    ("nine_impulses", 700)])
def test_gpu_1d_groups_match_oracle(kind, n):
    make, flights, half = MEDIA_1D[kind]
    desc = make()
    prim = flights(n, desc)
    with runtime.Context(desc) as ctx:
        rec_cpu, _ = flights_vs_oracle(desc, prim, ctx.trace_host(prim), scene=half)
        sec, _ = workloads.secondary_flights(prim, rec_cpu, desc, half=half)
        if sec.n:
            flights_vs_oracle(desc, sec, ctx.trace_host(sec), scene=half)


@pytest.mark.parametrize("precise", [0, 1])
def test_gpu_1d_group_and_lane_passes_agree(precise):
    """The resume passes on groups and on single lanes decide the same bits: a batch whose
    queue is longer than the limit against the same flights in batches below it."""
    desc = workloads.sphere_medium()
    prim = workloads.sphere_flights(300_000, desc)
    with runtime.Context(desc) as ctx:
        ctx.tune(abi.TUNE_PRECISE_DECISIONS, precise)
        whole = ctx.trace_host(prim)
        parts = [ctx.trace_host(prim.subset(np.arange(k, k + 50_000))) for k in range(0, prim.n, 50_000)]
    part = np.concatenate(parts)
    hit = abi.unpack_results(whole)["hit"]
    assert hit.sum() > 200_000
    assert np.array_equal(whole[hit].view(np.uint32), part[hit].view(np.uint32))
    a, b = abi.unpack_results(whole), abi.unpack_results(part)
    for name in ("status", "steps", "hit", "t", "gp_id"):
        assert np.array_equal(a[name], b[name]), name
    assert np.abs(a["value"] - b["value"]).max() <= 2e-6
