"""The forms of a pass that only long queues or device-side counts take: records and images
do not depend on which form decided a flight."""
import numpy as np
import pytest

from gpis_extend_gb300 import abi, workloads
from test_lane_groups import MEDIA_1D, sphere_grid_stationary

pytestmark = pytest.mark.gpu


def parts(ctx, prim, n):
    return np.concatenate([ctx.trace_host(prim.subset(np.arange(k, min(k + n, prim.n)))) for k in range(0, prim.n, n)])


def test_gpu_grid_groups_and_lanes_agree():
    """A grid mean: eight lanes a flight below 32 000 flights, one above."""
    from gpis_extend_gb300 import runtime
    desc = sphere_grid_stationary()
    prim = workloads.sphere_flights(48_000, desc)
    with runtime.Context(desc) as ctx:
        whole = ctx.trace_host(prim)
        groups = parts(ctx, prim, 16_000)
        sec, _ = workloads.secondary_flights(prim, whole, desc)
        two = abi.FlightBatch(2 * sec.n)
        for name in ("origin_near", "dir_far", "seeds", "prev"):
            getattr(two, name)[:] = np.concatenate([getattr(sec, name)] * 2)
        whole2 = ctx.trace_host(two)
        groups2 = parts(ctx, sec, 16_000)
    assert np.array_equal(whole.view(np.uint32), groups.view(np.uint32))
    assert two.n > 32_000 and np.array_equal(whole2[:sec.n].view(np.uint32), groups2.view(np.uint32))


@pytest.mark.parametrize("kind,n", [("octaves", 130_000), ("multires", 130_000), ("nonstationary", 130_000),
                                    ("nonstationary", 1_150_000)])
def test_gpu_precise_forms_agree(kind, n):
    """Precise passes of general media: a warp a flight below 60 000 queued flights, eight
    lanes below 1 000 000, one above."""
    from gpis_extend_gb300 import runtime
    make, flights, _ = MEDIA_1D[kind]
    desc = make()
    prim = flights(n, desc)
    with runtime.Context(desc) as ctx:
        whole = ctx.trace_host(prim)
        assert abi.unpack_results(whole)["hit"].sum() > (1_000_000 if n > 1_000_000 else 60_000)
        few = parts(ctx, prim, 40_000)
    assert np.array_equal(whole.view(np.uint32), few.view(np.uint32))


@pytest.mark.parametrize("kind,size,passes", [("torus", (96, 96, 4), (9216, 18_432)),
                                              ("sphere_1d", (160, 160, 2), (25_600,)),
                                              ("sphere_3d", (96, 96, 2), (9216,))])
def test_gpu_live_counts_on_both_sides_of_the_lines(kind, size, passes):
    """Batches whose length is known on the device only, on both sides of the lines between
    the forms (12 000, 20 000 and 32 000 flights in 1D, 10 000 in 3D): a render in passes of
    other sizes is the same image.  A pass holds whole samples of the image."""
    from gpis_extend_gb300 import runtime
    w, h, spp = size
    scene = workloads.render_scene(width=w, height=h, spp=spp, max_bounces=2, box_half=2.0 if kind == "torus" else 1.5)
    with runtime.Context(workloads.render_medium(kind)) as ctx:
        ref, st = ctx.render(scene)
        assert st["passes"] == 1
        for p in passes:
            ctx.tune(abi.TUNE_RENDER_PASS_PATHS, p)
            got, st = ctx.render(scene)
            assert st["passes"] > 1 and np.array_equal(ref, got), p
