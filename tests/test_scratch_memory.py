"""The scratch that a context holds per flight of its largest batch: 176 bytes bound the
largest batch that fits before octave, nonstationary and multi-resolution media took set-up
records, and still do."""
import pytest

from gpis_extend_gb300 import abi, workloads
from test_lane_groups import MEDIA_1D


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["sphere", "octaves", "multires", "nonstationary", "nine_impulses", "3d"])
def test_gpu_scratch_per_flight(kind):
    torch = pytest.importorskip("torch")
    from gpis_extend_gb300 import runtime
    if kind == "3d":
        make, flights = (lambda: workloads.sphere_medium(one_d=False)), workloads.sphere_flights
    else:
        make, flights, _ = MEDIA_1D[kind]
    desc = make()
    n = 1 << 20
    with runtime.Context(desc) as ctx:
        small = runtime.DeviceFlights(flights(1024, desc))
        ctx.submit(small)                   # (modules and the context's own, before the batch's)
        torch.cuda.synchronize()
        # rays that miss the field's box: short, for the scratch alone
        b = abi.FlightBatch(n)
        for name in ("origin_near", "dir_far", "seeds", "prev"):
            getattr(b, name)[:] = getattr(flights(1, desc), name)[0]
        b.dir_far[:, 3] = 0.01
        dev = runtime.DeviceFlights(b)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        ctx.submit(dev)
        torch.cuda.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
    print(kind, "bytes a flight", used / n)
    # five buffers, each rounded up to 2 MiB
    assert used <= 176 * n + 5 * (2 << 20)
