"""gpis_counters.cell_refills counts the cells whose impulses were drawn, whatever evaluator
the batch's size takes.  A flight draws its first window (three cells an octave, 27 in 3D) at
least, and a window moves by a cell or stays, so an evaluation draws fewer than a window on
average.  The same flights in batches of another size draw the same windows in the fast
pass; the resume passes, a few evaluations a flight, may draw whole windows at each."""
import numpy as np
import pytest

from gpis_extend_gb300 import abi, workloads

pytestmark = pytest.mark.gpu

# name: medium, flights, the cells of a window, batch sizes (the last is the reference)
KINDS = {
    "sphere": (workloads.sphere_medium, workloads.sphere_flights, 3, (8000, 40_000)),
    "octaves": (workloads.torus_plane_medium, workloads.torus_flights, 9, (8000, 16_000, 48_000)),
    "multires": (lambda: workloads.torus_plane_medium(octaves=1, multires=1), workloads.torus_flights, 6,
                 (8000, 16_000, 48_000)),
    "nonstationary": (lambda: workloads.torus_plane_medium(octaves=1), workloads.torus_flights, 3,
                      (8000, 16_000, 48_000)),
    "3d": (lambda: workloads.sphere_medium(one_d=False, impulse_density=8.0), workloads.sphere_flights, 27,
           (8000, 24_000)),
}


@pytest.mark.parametrize("kind", KINDS)
def test_gpu_refills_count_drawn_cells(kind):
    from gpis_extend_gb300 import runtime
    make, flights, window, sizes = KINDS[kind]
    desc = make()
    prim = flights(sizes[-1], desc)
    per = {}
    with runtime.Context(desc) as ctx:
        for n in sizes:
            ctx.counters(reset=True)
            for k in range(0, prim.n, n):
                ctx.trace_host(prim.subset(np.arange(k, k + n)))
            c = ctx.counters(reset=True)
            assert c["flights"] == prim.n
            evals = c["steps"] - c["skipped_steps"] + c["refine_evals"] + c["flights"]
            per[n] = c["cell_refills"] / prim.n
            print(kind, n, "cells a flight", per[n], "evaluations a flight", evals / prim.n)
            assert window <= per[n] <= window * evals / prim.n
    for n in sizes[:-1]:
        assert 0.5 <= per[n] / per[sizes[-1]] <= 2.0, per
