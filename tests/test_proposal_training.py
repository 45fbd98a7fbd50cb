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


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_gpu_features_at_block_edges(n):
    """The features kernel stores a block's 128 rows together: every row up to n (bar of
    test_gpu_features_match_restatement), nothing after the last."""
    torch = pytest.importorskip("torch")
    from gpis_extend_gb300 import runtime, workloads
    desc = proposal.config2_medium()
    b = workloads.torus_flights(n, desc)
    with runtime.Context(desc) as ctx:
        out = torch.full((n + 3, 24), 7.0, dtype=torch.float32, device="cuda")
        f = runtime.proposal_features(ctx, runtime.DeviceFlights(b), out=out).cpu().numpy()
    ref = R.features(desc, b.origin_near, b.dir_far, b.seeds, b.prev)
    assert np.all(np.abs(f[:n] - ref) <= 1e-4 * (1 + np.abs(ref)))
    assert np.all(f[n:] == 7.0)
