"""The reach before a proposed interval: a proposal costs no evaluations where its interval is
right, and GPIS_TUNE_PROPOSED_SKIP_CAP is the limit it is documented as.  The records are the
plain ones whatever the intervals and the limit."""
import numpy as np
import pytest

from gpis_extend_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

MEDIA = {
    "sphere": (workloads.sphere_medium, workloads.sphere_flights),
    "octaves": (workloads.torus_plane_medium, workloads.torus_flights),
    "nonstationary": (lambda: workloads.torus_plane_medium(octaves=1), workloads.torus_flights),
    "multires": (lambda: workloads.torus_plane_medium(octaves=1, multires=1), workloads.torus_flights),
}


def run(ctx, dev, intervals):
    import torch
    from gpis_extend_gb300 import runtime
    dev.rec.zero_()
    ctx.counters(reset=True)
    if intervals is None:
        ctx.submit(dev)
    else:
        runtime.submit_proposed(ctx, dev, intervals)
    torch.cuda.synchronize()
    c = ctx.counters(reset=True)
    return dev.rec.cpu().numpy().copy(), c["steps"] - c["skipped_steps"]


@pytest.mark.parametrize("n", [2000, 16_000, 40_000])
@pytest.mark.parametrize("kind", MEDIA)
def test_gpu_true_interval_costs_no_evaluations(kind, n):
    """The true crossing as the interval, and none (the whole flight lies before it): as many
    evaluations as without a proposal, at every limit from 64 steps."""
    import torch
    from gpis_extend_gb300 import runtime
    make, flights = MEDIA[kind]
    desc = make()
    prim = flights(n, desc)
    with runtime.Context(desc) as ctx:
        dev = runtime.DeviceFlights(prim)
        plain, evals = run(ctx, dev, None)
        r = abi.unpack_results(plain)
        far = prim.dir_far[:, 3]
        iv = np.zeros((n, 4), np.float32)
        iv[:, 0] = np.where(r["hit"], r["t"], far)
        iv[:, 1] = far
        last = iv.copy()
        last[:, 0] = far
        for cap in (0, 64, 256):
            ctx.tune(abi.TUNE_PROPOSED_SKIP_CAP, cap)
            for intervals in (iv, last):
                rec, got = run(ctx, dev, torch.from_numpy(intervals).cuda())
                print(kind, n, cap, got / n, evals / n)
                assert np.array_equal(rec.view(np.uint32), plain.view(np.uint32)), cap
                # (from 256 on a reach may be longer, and an evaluation ahead of the march
                # that lies beyond the crossing is one more: at most one a flight)
                assert got <= evals + (n if cap == 256 else 0), cap


@pytest.mark.parametrize("kind", MEDIA)
def test_gpu_skip_cap_limits_the_reach(kind):
    """Limits below the march's own take effect.  On a plain medium a lower one means more
    evaluations; elsewhere the bound is taken over the span, and a shorter span may serve
    better."""
    import torch
    from gpis_extend_gb300 import runtime
    make, flights = MEDIA[kind]
    desc = make(step_size=0.002) if kind == "sphere" else make()
    prim = flights(16_000, desc)
    iv = np.zeros((prim.n, 4), np.float32)
    iv[:, 0] = iv[:, 1] = prim.dir_far[:, 3]
    with runtime.Context(desc) as ctx:
        dev = runtime.DeviceFlights(prim)
        ivd = torch.from_numpy(iv).cuda()
        plain, evals = run(ctx, dev, None)
        seen = []
        for cap in (8, 16, 64):
            ctx.tune(abi.TUNE_PROPOSED_SKIP_CAP, cap)
            rec, got = run(ctx, dev, ivd)
            assert np.array_equal(rec.view(np.uint32), plain.view(np.uint32)), cap
            seen.append(got)
        print(kind, [s / prim.n for s in seen], evals / prim.n)
        assert seen[2] <= evals
        if kind == "sphere":
            assert seen[0] > seen[1] > seen[2]
        else:
            assert len(set(seen)) == 3
