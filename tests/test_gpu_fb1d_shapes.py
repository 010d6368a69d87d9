"""phmm_fb1d at the sizes where its shapes change: states around the vector bounds (8, 20, 32, 44, 64) and columns
around the counting batches (8 a warp, 4 or 8 warps) and the load-ahead of 4, with dense emissions, one-type emissions
and an impossible alignment, against the float64 oracle.  Bars of the float32 recursion as elsewhere: log P 1e-6
relative, posteriors 1e-5 absolute, expected transitions 1e-5 of the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LENGTHS = [1, 2, 3, 4, 5, 8, 9, 31, 32, 33, 63, 64, 65, 66, 130]


@pytest.mark.parametrize('n', [2, 5, 8, 9, 20, 21, 32, 33, 44, 45, 64])
@pytest.mark.parametrize('dense', [True, False])
def test_shapes_match_oracle(cuda_lib, n, dense):
    from pairhmm import api
    from oracle import fb1d
    rng = np.random.default_rng(100 * n + dense)
    chi = rng.dirichlet(np.ones(n), n) * 0.98
    chi[rng.random((n, n)) < 0.2] = 0.0
    chi[0, :] = 1.0 / n
    init, final = 0, n - 1
    chi[:, final] = np.maximum(chi[:, final], 0.01)
    em = rng.uniform(1e-3, 0.2, (len(LENGTHS) + 1, max(LENGTHS), n))
    if not dense:   # a column emits through the states of one residue class
        kind = rng.integers(0, 2, (len(LENGTHS) + 1, max(LENGTHS)))
        em = em * ((np.arange(n) % 2)[None, None, :] == kind[..., None])
        chi = np.maximum(chi, 0.001)
    lens = LENGTHS + [12]
    em[-1, 7] = 0.0   # impossible
    log = lambda v: np.where(v > 0, np.log(np.maximum(v, 1e-300)), -1e30)
    lp, post, nt = api.forward_backward_1d_batch(log(chi), log(em), lens, init, final)
    for b, L in enumerate(LENGTHS):
        want, wpost, wn = fb1d.forward_backward_1d(log(chi), log(em[b, :L]), init, final)
        assert abs(lp[b].item() - want) <= 1e-6 * abs(want), L
        np.testing.assert_allclose(post[b, :L].cpu().numpy(), wpost, atol=1e-5)
        assert np.abs(nt[b].cpu().numpy() - wn).max() <= 1e-5 * np.abs(wn).max(), L
    assert lp[-1].item() == -1e30 and float(nt[-1].abs().max()) == 0.0
