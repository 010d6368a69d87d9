"""The device emission tables of the gradient path (phmm_mixdom2_emissions, _vjp) against automatic differentiation of
the float64 tensor builders on the CPU, and phmm_fb1d_counts against summed posteriors: one to eight classes, more groups
than warps, times on both sides of the exponential's degree and scaling bounds, zero class weights, residues at the
wildcard.  Float64 on both sides; the exponential's derivative accumulates at most a few hundred roundings of entries
bounded by the largest, so 1e-11 of the largest gradient."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('K,F,C,P', [(1, 1, 1, 1), (3, 1, 1, 5), (4, 2, 2, 3), (2, 1, 8, 2), (8, 4, 4, 2)])
def test_tables_and_gradients(cuda_lib, K, F, C, P):
    from pairhmm import _lib, api, synth
    from pairhmm import models as pm
    rng = np.random.default_rng(K * 100 + C)
    p = synth.mixdom2_params(rng, K, F, C)
    if C > 1:
        p['classdist'][0, 0] = np.eye(C)[1]
    ts = np.concatenate([[0.02, 0.2, 0.7, 3.0, 30.0][:P]])
    keys = ('class_S_exch', 'class_pis', 'classdist')
    leaf = lambda dev: [torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True)
                        for v in [ts] + [p[k] for k in keys]]
    G = K * F
    wM, wI, wD = (torch.tensor(rng.normal(size=s)) for s in ((P, G, 21, 21), (P, G, 21), (P, G, 21)))
    a = leaf('cpu')
    EM, EI, ED = pm.tables_per_class(pm.class_subs(a[1], a[2], a[0]), a[2], a[3])
    ((EM * wM).sum() + (EI * wI).sum() + (ED * wD).sum()).backward()
    b = leaf('cuda')
    dM, dI = api.MixDom2Emissions.apply(_lib.MixDom2Prologue(p), *b)
    ((dM * wM.cuda()).sum() + (dI * wI.cuda()).sum() + (dI * wD.cuda()).sum()).backward()
    for got, want in ((dM, EM), (dI, EI.expand(P, G, 21))):
        assert (got.detach().cpu() - want.detach()).abs().max() <= 1e-13
    for x, y in zip(a, b):
        assert y.grad.shape == x.grad.shape
        assert (y.grad.cpu() - x.grad).abs().max() <= 1e-11 * x.grad.abs().max()


@pytest.mark.parametrize('n', [5, 32, 33, 62])
def test_alignment_counts(cuda_lib, n):
    from pairhmm import _lib
    rng = np.random.default_rng(n)
    lens = [0, 1, 7, 8, 9, 300]
    off = np.concatenate([[0], np.cumsum(lens)[:-1]])
    total, G = sum(lens), 3
    st = np.concatenate([[0], rng.integers(1, 4, n - 2), [4]])
    gr = rng.integers(0, G, n)
    cols, anc, desc = (rng.integers(lo, hi, total).astype(np.uint8) for lo, hi in ((1, 4), (0, 22), (0, 22)))
    post = rng.random((total, n)).astype(np.float32)
    dev = lambda v: torch.from_numpy(v).cuda()
    got = _lib.fb1d_counts(st, gr, G, lens, off, dev(cols), dev(anc), dev(desc), dev(post))
    want = [np.zeros((len(lens), G, 21, 21)), np.zeros((len(lens), G, 21)), np.zeros((len(lens), G, 21))]
    for p, (o, L) in enumerate(zip(off, lens)):
        for l in range(o, o + L):
            x, y = min(anc[l], 20), min(desc[l], 20)
            for s in np.nonzero(st == cols[l])[0]:
                at = {1: (p, gr[s], x, y), 2: (p, gr[s], y), 3: (p, gr[s], x)}[cols[l]]
                want[cols[l] - 1][at] += np.float64(post[l, s])
    for g, w in zip(got, want):
        np.testing.assert_allclose(g.cpu().numpy(), w, rtol=1e-13, atol=0)


@pytest.mark.parametrize('K,F', [(1, 1), (2, 3), (3, 1), (4, 2), (5, 1), (8, 4), (16, 2), (33, 1)])
def test_chi_gradients(cuda_lib, K, F):
    """One to 33 domains: every direction at once, several rounds of teams, one team (the bound of its other test, 1e-9)."""
    from pairhmm import _lib, api, synth
    from pairhmm import models as pm
    rng = np.random.default_rng(K * 10 + F)
    p = synth.mixdom2_params(rng, K, F, 1)
    p['ext_rates'] = rng.dirichlet(np.ones(F + 1), (K, F))[..., :F]      # a full fragment matrix
    keys = ('main_ins', 'main_del', 'dom_ins', 'dom_del', 'dom_weights', 'frag_weights', 'ext_rates')
    ts = np.array([0.3, 1.1])
    leaf = lambda dev: [torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True)
                        for v in [ts] + [p[k] for k in keys]]
    a, b = leaf('cpu'), leaf('cuda')
    chi = pm.build_nested_trans(a[1], a[2], a[0], *a[3:])
    w = torch.tensor(rng.normal(size=chi.shape))
    (chi * w).sum().backward()
    (api.MixDom2Chi.apply(_lib.MixDom2Prologue(p), *b) * w.cuda()).sum().backward()
    for x, y in zip(a, b):
        assert (y.grad.cpu() - x.grad).abs().max() <= 1e-9 * x.grad.abs().max()
