"""Stripes of 64 rows hand their boundary rows on word by word: the words of
one call must not be taken for those of the next.

The edge rows of a plan are reused by every call.  A plan that has run other
pairs (longer, and the same ones with other parameters) must give the
log-likelihood bits of a fresh plan, at lengths around the stripe height and at
the shortest rows, and without a mask both agree with the FP64 oracle within
the bounds of the other kernel tests (log-likelihood 1e-6, counts 1e-5 of the
largest: float32 recursion against float64)."""
import numpy as np
import pytest
import torch

from oracle import estep as oe, pool

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('masked', [False, True])
@pytest.mark.parametrize('K,F,C', [(1, 1, 1), (3, 1, 1), (4, 1, 2)])
@pytest.mark.parametrize('lens', [((64, 1), (65, 0), (1, 64), (128, 2)), ((127, 60), (191, 3), (192, 200), (63, 63))])
def test_reused_edge_rows(cuda_lib, K, F, C, lens, masked):
    from pairhmm import _lib, api, synth
    rng = np.random.default_rng(5)
    model = lambda: oe.mixdom2_model(synth.mixdom2_params(rng, K, F, C))[:6]
    (chi, st, groups, EM, EI, ED), other = model(), model()

    def batch(ls, tables):
        xs, ys = [rng.integers(0, 20, a) for a, _ in ls], [rng.integers(0, 20, b) for _, b in ls]
        m = [api.band_mask(a, b, np.round(np.arange(a + 1) * b / a).astype(int), 5) for a, b in ls] if masked else None
        return xs, ys, _lib.make_batch(xs, ys, *[t[None] for t in tables], device='cuda', cell_masks=m)

    tables = (chi, EM, EI, ED)
    others = (other[0],) + tuple(other[3:])
    used, fresh = _lib.Plan(st, groups, K * F), _lib.Plan(st, groups, K * F)
    _lib.estep(used, batch([(300, 310)] * 3, others)[2])
    _lib.estep(used, batch(lens, others)[2])
    xs, ys, b = batch(lens, tables)
    got, want = _lib.estep(used, b), _lib.estep(fresh, b)
    fwd = _lib.forward(used, b)[0], _lib.forward(fresh, b)[0]
    torch.cuda.synchronize()
    assert used.last_variant == 7
    assert torch.equal(got['status'], want['status']) and torch.equal(got['ll'], want['ll'])
    assert torch.equal(*fwd)
    if masked:
        return
    assert (got['status'] == 0).all()
    ref = pool.estep_pairs([(chi, st, groups, EM, EI, ED, x, y) for x, y in zip(xs, ys)])
    ll, n = got['ll'].cpu().numpy(), got['n_trans'].cpu().numpy()
    for k in range(len(xs)):
        assert abs(ll[k] - ref[k][0]) <= 1e-6 * abs(ref[k][0]) + 1e-9
        assert np.abs(n[k] - ref[k][1]).max() <= 1e-5 * np.abs(ref[k][1]).max()
