"""Band-layout posteriors and live column ranges at the edges of their loops:
pairs around the 64-row stripe, bands narrower and wider than a warp's 32
positions, mask rows at every alignment, 7 to 22 states, a pair without
likelihood -- against the dense posteriors of the generic kernels on the same
masks, within the bounds of the masked tests (relative 1e-5, absolute 1e-6:
two float32 recursions)."""
import numpy as np
import pytest
import torch

from oracle import estep as oe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('W', [0, 7, 40])
@pytest.mark.parametrize('K', [1, 3, 4])
def test_band_posteriors_match_dense(cuda_lib, K, W):
    from pairhmm import _lib, synth
    rng = np.random.default_rng(100 * K + W)
    chi, st, groups, EM, EI, ED, _ = oe.mixdom2_model(synth.mixdom2_params(rng, K, 1, 2))
    shapes = [(1, 1), (63, 70), (64, 64), (65, 49), (127, 128), (130, 14), (5, 200), (128, 113), (40, 40)]
    xs = [rng.integers(0, 20, a) for a, _ in shapes]
    ys = [rng.integers(0, 20, b) for _, b in shapes]
    centers = [np.round(np.arange(a + 1) * b / a).astype(int) for a, b in shapes]
    masks = [np.where(np.abs(np.arange(b + 1) - c[:, None]) <= W, 7, 0).astype(np.uint8)
             for (_, b), c in zip(shapes, centers)]
    masks[-1][20] = 0                                            # no path: no likelihood, all zero
    b = _lib.make_batch(xs, ys, chi[None], EM[None], EI[None], ED[None], device='cuda', cell_masks=masks)
    plan = _lib.Plan(st, groups, K)
    got = _lib.estep_band(plan, b, centers, W)
    ref = _lib.Plan(st, groups, K)
    ref.set_variant(1)
    want = _lib.estep_tables(ref, b, want_F=False, want_B=False)
    torch.cuda.synchronize()
    ll, wll = got['ll'].cpu().numpy(), want['ll'].cpu().numpy()
    post, band = want['post'].cpu().numpy().reshape(-1), got['post_band'].cpu().numpy()
    assert ll[-1] <= -1e29
    N, cell, row = chi.shape[0], 0, 0
    for k, (a, ly) in enumerate(shapes):
        dense = post[cell * N:(cell + (a + 1) * (ly + 1)) * N].reshape(a + 1, ly + 1, N)
        jj = centers[k][:, None] - W + np.arange(2 * W + 1)[None, :]
        expect = np.zeros((a + 1, 2 * W + 1, N))
        if wll[k] > -1e29:
            assert abs(ll[k] - wll[k]) <= 1e-6 * abs(wll[k])
            ii, bb = np.nonzero((jj >= 0) & (jj <= ly))
            expect[ii, bb] = dense[ii, jj[ii, bb]]
            expect[..., np.asarray(st) == 4] = 0.0               # the end state has no cell in band layout
        else:
            assert ll[k] <= -1e29
        np.testing.assert_allclose(band[row:row + a + 1], expect, rtol=1e-5, atol=1e-6)
        cell += (a + 1) * (ly + 1)
        row += a + 1
