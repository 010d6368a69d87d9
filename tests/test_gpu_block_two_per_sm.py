"""The 42-state block recursions at two CTAs an SM (more stripes than SMs) and at
one: the same pairs alone and among enough others, at lengths around the 64-row
stripe.  The recursions round alike (the same bits); the counts differ in the
order of the float64 additions only: 1e-12 of the largest."""
import numpy as np
import pytest
import torch

from oracle import estep as oe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('extra', [160, 320])   # stripes over the SMs for both directions; for the forward alone
def test_block_two_per_sm_matches_one(cuda_lib, extra):
    from pairhmm import _lib, synth
    rng = np.random.default_rng(extra)
    chi, st, groups, EM, EI, ED, _ = oe.mixdom2_model(synth.mixdom2_params(rng, 4, 2, 2))
    shapes = [(0, 2), (1, 0), (7, 3), (31, 32), (62, 5), (63, 63), (64, 1), (127, 66), (129, 20)]
    many = shapes + [(9, 8)] * extra
    xs = [rng.integers(0, 20, a) for a, _ in many]
    ys = [rng.integers(0, 20, b) for _, b in many]
    k = len(shapes)

    def run(n):
        plan = _lib.Plan(st, groups, 8)
        bt = _lib.make_batch(xs[:n], ys[:n], chi[None], EM[None], EI[None], ED[None], device='cuda')
        return _lib.estep(plan, bt), _lib.forward(plan, bt)[0]

    (got, gf), (want, wf) = run(len(many)), run(k)
    torch.cuda.synchronize()
    assert torch.equal(got['ll'][:k], want['ll']) and torch.equal(got['status'][:k], want['status'])
    assert torch.equal(gf[:k], wf)
    for n in ('n_trans', 'cnt_M', 'cnt_I', 'cnt_D'):
        a, b = got[n][:k].cpu().numpy(), want[n].cpu().numpy()
        for p in range(k):
            assert np.abs(a[p] - b[p]).max() <= 1e-12 * max(np.abs(b[p]).max(), 1e-300), (n, many[p])
