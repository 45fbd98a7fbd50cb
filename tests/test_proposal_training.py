"""The training gradient of the crossing proposal at the edges of its kernels' tiles
(128-flight GEMM tiles, 64-flight loss blocks, the K chunks of the weight gradients over
the rows of all steps): against the NumPy restatement, with the bar of
test_gpu_forward_and_gradient_match_reference (BF16 operands; relative L2 per tensor)."""
import numpy as np
import pytest

from gpis_extend_gb300 import proposal
from oracle import proposal_ref as R
from test_proposal import random_features, random_targets


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 48, 144, 1040, 5008])
def test_gpu_gradient_at_tile_edges(n):
    torch = pytest.importorskip("torch")
    from gpis_extend_gb300 import runtime
    rng = np.random.default_rng(n)
    f, tg = random_features(n, rng), random_targets(n, rng)
    params = proposal.init_params(7)
    with runtime.Proposal(params) as prop:
        fd, td = torch.from_numpy(f).cuda(), torch.from_numpy(tg).cuda()
        # a larger batch first, so that stale activations would show
        big = torch.from_numpy(random_features(2 * n + 32, rng)).cuda()
        prop.gradient(big, torch.from_numpy(random_targets(2 * n + 32, rng)).cuda())
        grad, loss = prop.gradient(fd, td)
    o, cache = R.forward(R.unflatten(params.astype(np.float64)), f)
    lref, g = R.loss_and_grad_out(o, tg[:, 0].astype(np.float64), tg[:, 1] > 0)
    gref = R.backward(R.unflatten(params.astype(np.float64)), cache, g)
    gd = R.unflatten(grad.astype(np.float64))
    assert abs(loss - lref) <= 1e-3 * (1 + abs(lref))
    for name, _ in R.PARAMS:
        rel = np.linalg.norm(gd[name] - gref[name]) / max(np.linalg.norm(gref[name]), 1e-12)
        assert rel <= 3e-2, (name, rel)
