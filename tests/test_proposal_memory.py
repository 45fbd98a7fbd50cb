"""The device memory of a training handle: 10.5 KB a flight bound the largest batch before
the GRU's weight gradients were taken over all steps at once, and still do."""
import numpy as np
import pytest

from gpis_extend_gb300 import proposal
from test_proposal import random_features, random_targets


@pytest.mark.gpu
def test_gpu_training_memory_per_flight():
    torch = pytest.importorskip("torch")
    from gpis_extend_gb300 import runtime
    n = 1 << 17
    rng = np.random.default_rng(3)
    with runtime.Proposal(proposal.init_params(1)) as prop:
        f = torch.from_numpy(random_features(n, rng)).cuda()
        t = torch.from_numpy(random_targets(n, rng)).cuda()
        prop.gradient(f[:16], t[:16])       # (the library's and the handle's own, before the batch's)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        prop.gradient(f, t)
        torch.cuda.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
    print("bytes a flight", used / n)
    # 24 buffers, each rounded up to 2 MiB
    assert used <= 10_528 * n + 24 * (2 << 20)
