"""phmm_tkf92_bdi, the TKF92 epilogue kernel, at batch sizes around its blocks: every pair's statistics must be those of
the pair alone, bit for bit (their values are checked through estep_batch_tkf92 in test_gpu_api_golden.py)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def counts(rng, P):
    n = rng.uniform(0.0, 3.0, (P, 5, 5))
    n[:, :, 0] = 0.0        # nothing enters the start state
    n[:, 4, :] = 0.0        # nothing leaves the end state
    return n


@pytest.mark.parametrize('P', [1, 31, 32, 33, 70])
def test_block_edges(cuda_lib, P):
    from pairhmm import bdi
    rng = np.random.default_rng(P)
    n, t = counts(rng, P), np.exp(rng.uniform(np.log(1e-3), np.log(30.0), P))
    n[P // 2] = 0.0
    got = bdi.tkf92_bdi_epilogue(torch.tensor(n).cuda(), 0.03, 0.04, t, 0.5)
    for b in range(P):
        one = bdi.tkf92_bdi_epilogue(torch.tensor(n[b:b + 1]).cuda(), 0.03, 0.04, t[b:b + 1], 0.5)
        for k in got:
            assert torch.equal(got[k][b], one[k][0]), (k, b)


def test_differentiated_and_equal_rate_counts_take_the_tensor_form(cuda_lib):
    from pairhmm import bdi
    n = torch.rand(3, 5, 5, dtype=torch.float64).cuda()
    a = bdi.tkf92_bdi_epilogue(n.clone().requires_grad_(), 0.03, 0.04, np.ones(3), 0.5)
    assert a['L'].requires_grad
    b = bdi.tkf92_bdi_epilogue(n, 0.03, 0.03, np.ones(3), 0.5)
    assert all(bool(torch.isfinite(v).all()) for v in b.values())
