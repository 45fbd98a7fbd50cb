"""Votes among lanes.  The groups of a warp diverge from one another, and only a mask that
is fixed by the program says which lanes take part in a vote or a shuffle: the set of
lanes that happen to be converged decides nothing."""
import os
import re

import numpy as np
import pytest

from gpis_extend_gb300 import abi, build, workloads


def test_votes_name_their_lanes():
    for name in sorted(os.listdir(build.CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(build.CSRC, name)) as f:
            code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
        assert "__activemask" not in code, name


@pytest.mark.gpu
def test_gpu_3d_groups_in_unlike_phases():
    """Eight lanes a flight, four flights a warp, neighbours of unequal length and distance
    from the surface, so that at most iterations some of a warp's flights plan a range and
    others do not: the records of a warp per flight, which votes with itself alone."""
    from gpis_extend_gb300 import runtime
    desc = workloads.sphere_medium(one_d=False, impulse_density=8.0, context=abi.CTX_RENEWAL)
    prim = workloads.sphere_flights(12_000, desc)
    far = prim.dir_far[:, 3].copy()
    prim.dir_far[1::4, 3] = np.float32(0.3) * far[1::4]
    prim.dir_far[2::4, 3] = np.float32(0.02) * far[2::4]
    prim.origin_near[3::4, 3] = np.float32(0.5) * far[3::4]
    with runtime.Context(desc) as ctx:
        many = ctx.trace_host(prim)
        few = np.concatenate([ctx.trace_host(prim.subset(np.arange(k, k + 4000))) for k in range(0, prim.n, 4000)])
        sec, _ = workloads.secondary_flights(prim, many, desc)
        two = abi.FlightBatch(3 * sec.n)
        for name in ("origin_near", "dir_far", "seeds", "prev"):
            getattr(two, name)[:] = np.concatenate([getattr(sec, name)] * 3)
        many2 = ctx.trace_host(two)
        few2 = ctx.trace_host(sec)
    assert np.array_equal(many.view(np.uint32), few.view(np.uint32))
    assert sec.n < 10_000 < two.n
    assert np.array_equal(many2.view(np.uint32), np.concatenate([few2] * 3).view(np.uint32))
