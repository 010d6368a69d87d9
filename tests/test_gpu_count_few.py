"""The count pass of few chunks against the count pass of many: the same pairs
alone and among enough others that their chunks outnumber the SMs, at lengths
around the 64-row stripe, the 64-step chunk and the four steps of a round, with
and without a mask.  Both add the same float terms in the same order and differ
in the order of the float64 additions only: 1e-12 of the largest count."""
import numpy as np
import pytest
import torch

from oracle import estep as oe

pytestmark = pytest.mark.gpu
NAMES = ('n_trans', 'cnt_M', 'cnt_I', 'cnt_D')


@pytest.mark.parametrize('masked', [False, True])
@pytest.mark.parametrize('K', [0, 1, 2, 3, 4])
def test_few_chunks_match_many(cuda_lib, K, masked):
    from pairhmm import _lib, synth
    rng = np.random.default_rng(K)
    if K:
        chi, st, groups, EM, EI, ED, _ = oe.mixdom2_model(synth.mixdom2_params(rng, K, 1, 2))
        G = K
    else:
        q = synth.tkf_params(rng, ext=0.5)
        chi, EM, EI, ED, _ = _lib.tkf92_tables(q['ins_rate'], q['del_rate'], 0.5, q['Q'], q['pi'], np.full(1, 0.5))
        chi, EM, EI, ED = (t[0].cpu().numpy() for t in (chi, EM, EI, ED))
        st, groups, G = np.array([0, 1, 2, 3, 4], np.int8), np.zeros(5, np.int32), 1
    shapes = [(0, 3), (1, 1), (3, 0), (5, 62), (63, 1), (64, 64), (65, 66), (40, 127), (130, 5)]
    many = shapes + [(200, 210)] * 16                       # 16 x 4 stripes x 5 chunks and more
    xs = [rng.integers(0, 20, a) for a, _ in many]
    ys = [rng.integers(0, 20, b) for _, b in many]

    def run(n):
        m = [np.where(np.abs(np.arange(b + 1) - np.arange(a + 1)[:, None] * b / max(a, 1)) <= 9, 7, 0).astype(np.uint8)
             for a, b in many[:n]] if masked else None
        bt = _lib.make_batch(xs[:n], ys[:n], chi[None], EM[None], EI[None], ED[None], device='cuda', cell_masks=m)
        return _lib.estep(_lib.Plan(st, groups, G), bt)

    got, want = run(len(shapes)), run(len(many))
    torch.cuda.synchronize()
    k = len(shapes)
    assert torch.equal(got['ll'], want['ll'][:k]) and torch.equal(got['status'], want['status'][:k])
    for n in NAMES:
        a, b = got[n].cpu().numpy(), want[n][:k].cpu().numpy()
        for p in range(k):
            assert np.abs(a[p] - b[p]).max() <= 1e-12 * max(np.abs(b[p]).max(), 1e-300), (n, many[p])
