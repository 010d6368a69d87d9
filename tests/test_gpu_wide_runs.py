"""The wide count pass in runs of a stripe's steps (few stripes) and whole (many):
the same 162-state pairs alone and among enough others, at lengths around the
32-row stripe and the 96-step least run.  The recursions add their type sums in no
fixed order and the partial sums are float32, so the bound is the other kernel
tests': counts 1e-5 of the largest."""
import numpy as np
import pytest
import torch

from oracle import estep as oe

pytestmark = pytest.mark.gpu


def test_wide_runs_match_whole(cuda_lib):
    from pairhmm import _lib, synth
    rng = np.random.default_rng(3)
    chi, st, groups, EM, EI, ED, _ = oe.mixdom2_model(synth.mixdom2_params(rng, 8, 4, 4))
    shapes = [(31, 64), (32, 65), (1, 95), (0, 96), (20, 175), (33, 193), (5, 3)]
    many = shapes + [(2, 3)] * 460                     # 920 half-stripes and more
    xs = [rng.integers(0, 20, a) for a, _ in many]
    ys = [rng.integers(0, 20, b) for _, b in many]
    k = len(shapes)

    def run(n):
        bt = _lib.make_batch(xs[:n], ys[:n], chi[None], EM[None], EI[None], ED[None], device='cuda')
        return _lib.estep(_lib.Plan(st, groups, 32), bt)

    got, want = run(k), run(len(many))
    torch.cuda.synchronize()
    assert (got['status'] == 0).all() and (want['status'] == 0).all()
    for n in ('n_trans', 'cnt_M', 'cnt_I', 'cnt_D'):
        a, b = got[n].cpu().numpy(), want[n][:k].cpu().numpy()
        for p in range(k):
            assert np.abs(a[p] - b[p]).max() <= 1e-5 * max(np.abs(b[p]).max(), 1e-300), (n, many[p])
