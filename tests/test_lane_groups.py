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
from test_skipping import sphere_grid

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
    """Both group sizes on the same flights give the same records."""
    desc = medium_3d(8, context=abi.CTX_RENEWAL)
    prim = workloads.sphere_flights(10500, desc)
    idx = np.arange(0, prim.n, 3)
    with runtime.Context(desc) as ctx:
        many = ctx.trace_host(prim)[idx]
        few = ctx.trace_host(prim.subset(idx))
    assert np.array_equal(many.view(np.uint32), few.view(np.uint32))


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
    assert abi.unpack_results(whole)["hit"].sum() > 200_000
    assert np.array_equal(whole.view(np.uint32), part.view(np.uint32))


@pytest.mark.parametrize("kind", ["sphere", "octaves", "multires", "nonstationary", "xy"])
def test_gpu_1d_fast_passes_agree(kind):
    """The fast passes on groups and on single lanes give the same records (misses too)."""
    make, flights, half = MEDIA_1D[kind]
    desc = make()
    prim = flights(48_000, desc)
    with runtime.Context(desc) as ctx:
        whole = ctx.trace_host(prim)
        # 6 000: a warp per flight in media of several octaves, 16 000: eight lanes
        parts = np.concatenate([ctx.trace_host(prim.subset(np.arange(k, k + 6000))) for k in range(0, prim.n, 6000)])
        eights = np.concatenate([ctx.trace_host(prim.subset(np.arange(k, k + 16000))) for k in range(0, prim.n, 16000)])
        sec, _ = workloads.secondary_flights(prim, whole, desc, half=half)
        two = abi.FlightBatch(2 * sec.n)
        for name in ("origin_near", "dir_far", "seeds", "prev"):
            getattr(two, name)[:] = np.concatenate([getattr(sec, name)] * 2)
        whole2 = ctx.trace_host(two)
        parts2 = np.concatenate([ctx.trace_host(sec.subset(np.arange(k, min(k + 6000, sec.n))))
                                 for k in range(0, sec.n, 6000)])
    assert np.array_equal(whole.view(np.uint32), parts.view(np.uint32))
    assert np.array_equal(whole.view(np.uint32), eights.view(np.uint32))
    assert two.n > 45_000 and np.array_equal(whole2[:sec.n].view(np.uint32), parts2.view(np.uint32))


def sphere_grid_stationary():
    return abi.attach_grid(workloads.sphere_medium(), sphere_grid())


def torus_stationary(**kw):
    return workloads.torus_plane_medium(nonstationary=False, octaves=1, **kw)


@pytest.mark.parametrize("kind,n", [("octaves", 45001), ("multires", 45001), ("nonstationary", 46000), ("sphere", 40001),
                                    ("torus", 40961), ("plane", 41003), ("grid", 40500)])
def test_gpu_1d_lane_passes_match_oracle(kind, n):
    """Batches just above the limits of the group fast passes: the cooperative single-lane
    passes, whose evaluations decide steps on both sides (the slope bound of several
    octaves, of a nonstationary scale and of the multi-resolution grid; the second-order
    reach of stationary media with a sphere, torus and linear mean)."""
    if kind == "torus":
        make, flights, half = torus_stationary, workloads.torus_flights, 2.0
    elif kind == "grid":
        make, flights, half = sphere_grid_stationary, workloads.sphere_flights, 1.5
    elif kind == "plane":
        make = lambda: workloads.sphere_medium(mean_kind=abi.MEAN_PLANE, mean_params=(0.0, 0.8, 0.6, 0.1))
        flights, half = workloads.sphere_flights, 1.5
    else:
        make, flights, half = MEDIA_1D[kind]
    desc = make()
    prim = flights(n, desc)
    with runtime.Context(desc) as ctx:
        ctx.counters(reset=True)
        rec = ctx.trace_host(prim)
        cnt = ctx.counters(reset=True)
        assert cnt["skipped_steps"] > 0.2 * cnt["steps"], cnt
        rec_cpu, _ = flights_vs_oracle(desc, prim, rec, scene=half)
        steps_gpu, steps_cpu = abi.unpack_results(rec)["steps"], abi.unpack_results(rec_cpu)["steps"]
        assert np.mean(steps_gpu == steps_cpu) >= 0.9999
        sec, _ = workloads.secondary_flights(prim, rec_cpu, desc, half=half)
        if sec.n > 45000 or kind in ("sphere", "torus", "plane"):
            flights_vs_oracle(desc, sec, ctx.trace_host(sec), scene=half)


@pytest.mark.parametrize("far,step,max_steps", [(0.004, 0.01, 0), (3.0, 0.01, 37), (3.0, 0.75, 0), (3.0, 0.01, 300)])
def test_gpu_reach_ends_with_the_march(far, step, max_steps):
    """Reaches that pass farT or the step limit: the steps taken and the statuses are the
    oracle's (flights shorter than a step, a limit inside the first reach, coarse steps)."""
    desc = workloads.sphere_medium(step_size=step, min_step=1, max_steps=max_steps)
    prim = workloads.sphere_flights(3000, desc)
    prim.dir_far[:, 3] = np.minimum(prim.dir_far[:, 3], np.float32(far))
    prim.dir_far[::7, 3] *= np.float32(0.37)
    rec_cpu = oracle.trace_flights(desc, prim)
    c = abi.unpack_results(rec_cpu)
    with runtime.Context(desc) as ctx:
        g = abi.unpack_results(ctx.trace_host(prim))
    assert np.array_equal(g["status"], c["status"])
    assert np.array_equal(g["steps"], c["steps"])
    assert np.array_equal(g["hit"], c["hit"])
    many = abi.FlightBatch(45_000)
    idx = np.arange(45_000) % 3000
    for name in ("origin_near", "dir_far", "seeds", "prev"):
        getattr(many, name)[:] = getattr(prim, name)[idx]
    with runtime.Context(desc) as ctx:
        g = abi.unpack_results(ctx.trace_host(many))
    assert np.array_equal(g["status"], c["status"][idx])
    assert np.array_equal(g["steps"], c["steps"][idx])
    assert np.array_equal(g["hit"], c["hit"][idx])


@pytest.mark.parametrize("kind,n", [("sphere", 3000), ("sphere", 40000), ("octaves", 2500), ("octaves", 24000),
                                    ("multires", 24000)])
def test_gpu_crossing_within_the_last_partial_step(kind, n):
    """farT just behind a crossing, which then lies in the last partial step: the march ends
    without it and the value at farT has the other sign."""
    make, flights, half = MEDIA_1D[kind]
    desc = make()
    prim = flights(n, desc)
    with runtime.Context(desc) as ctx:
        r = abi.unpack_results(ctx.trace_host(prim))
        hit = r["hit"] & (r["t"] > 0.0)
        step = np.minimum(np.float32(desc.step_size), prim.dir_far[:, 3] / np.float32(desc.min_step))
        cut = hit & (np.arange(n) % 4 != 0)
        prim.dir_far[cut, 3] = r["t"][cut] + np.float32(0.25) * step[cut]
        rec = ctx.trace_host(prim)
        rec_cpu, _ = flights_vs_oracle(desc, prim, rec, scene=half)
    g, c = abi.unpack_results(rec), abi.unpack_results(rec_cpu)
    miss = ~c["hit"] & ~g["hit"] & cut
    assert miss.sum() > 0.2 * cut.sum()
    assert np.array_equal(g["steps"][miss], c["steps"][miss])
    # the oracle's float formulation and the fast value differ by a few 1e-8 of the noise;
    # a truncation edge between the two roundings of the point moves it by at most 6e-4
    off = np.abs(g["value"][miss] - c["value"][miss])
    assert np.mean(off <= 2e-6) >= 0.999 and off.max() <= 2e-3
