"""gpis_render_stats.launches: the kernels a render launches, the passes of its flight batches
one by one.  A round launches advance, event, shadow, collect and tally around a distance
and a shadow batch of up to n and 2 n flights (n paths a pass); the batches' lengths are
known on the device only, so every form of a pass that their capacity allows is launched."""
import pytest

from gpis_extend_gb300 import workloads

pytestmark = pytest.mark.gpu

# per batch: prepare and finish, then the passes' forms by capacity
CASES = [
    # plain 1D: fast, certified and precise pass on groups
    ("sphere_1d", (32, 32, 1), 5, 5),
    # ... from 32 000 flights also the lanes' fast pass and its tail, from 100 000 the
    # lanes' certified pass
    ("sphere_1d", (256, 256, 1), 7, 8),
    # octaves: a warp per flight in the fast and the precise pass
    ("torus", (32, 32, 1), 4, 4),
    # ... from 12 000 eight lanes too, from 20 000 the lanes and the tail in both group
    # sizes, from 60 000 the precise pass in eights
    ("torus", (128, 128, 2), 8, 9),
    # 3D: one fast kernel for both group sizes, one resume pass
    ("sphere_3d", (32, 32, 1), 4, 4),
]


@pytest.mark.parametrize("profile", [False, True])
@pytest.mark.parametrize("kind,size,distance,shadow", CASES)
def test_gpu_render_counts_its_launches(kind, size, distance, shadow, profile):
    """As a captured graph and as direct launches (profiling on)."""
    from gpis_extend_gb300 import runtime
    w, h, spp = size
    bounces = 1
    scene = workloads.render_scene(width=w, height=h, spp=spp, max_bounces=bounces,
                                   box_half=2.0 if kind == "torus" else 1.5)
    with runtime.Context(workloads.render_medium(kind)) as ctx:
        ctx.profile(profile)
        _, st = ctx.render(scene)
    assert st["graphed"] == (0 if profile else 1) and st["passes"] == 1
    rounds = 2 * bounces + 4
    # a shadow batch before the first round sizes the scratch; camera, accumulate, finish
    assert st["launches"] == shadow + 3 + rounds * (5 + distance + shadow), st
