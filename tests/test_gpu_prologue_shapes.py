"""The prologue's matrix exponential and the class split where their paths change, against float64 references.

exp(tQ): 1-norms around the polynomial's degree and scaling bounds (0.06, 0.3, 0.7 and its doublings), zero time and
long times, reversible and general rate matrices, against scipy's Pade form.  Rows sum to one and entries are at most
one, so each of up to ten squarings adds at most about 20 roundings: 20 * 10 * 2^-53 * 4 < 1e-13.

Class split: batch sizes on each side of the column split (P * parts * 2 <= 304), more groups than warps, one to eight
classes, zero counts and class weights, against the tensor form of pairhmm.api.class_split on the CPU; sums of at most 32
groups or 483 columns of positive terms: 500 * 2^-53 * 4 < 1e-12 relative to the pair's largest."""
import numpy as np
import pytest
import scipy.linalg
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('general', [False, True])
def test_expm_at_its_bounds(cuda_lib, general):
    from pairhmm import _lib, synth
    rng = np.random.default_rng(1)
    Q, pi, _ = synth.rand_Q_pi(rng)
    if general:
        Q = rng.lognormal(0.0, 1.5, (20, 20))
        np.fill_diagonal(Q, 0.0)
        np.fill_diagonal(Q, -Q.sum(axis=1))
    norm = np.abs(Q).sum(axis=0).max()
    at = [0.06, 0.3, 0.7, 1.4, 2.8, 5.6, 22.4, 300.0]
    ts = np.array([0.0, 1e-6 / norm] + [v * f / norm for v in at for f in (1 - 1e-9, 1.0, 1 + 1e-9, 1.3)])
    sub = _lib.tkf92_tables(0.03, 0.04, 0.5, Q, pi, ts)[4].cpu().numpy()
    for t, got in zip(ts, sub):
        assert np.abs(got - scipy.linalg.expm(t * Q)).max() <= 1e-13, t * norm


@pytest.mark.parametrize('P', [1, 9, 76, 77, 152, 153])
@pytest.mark.parametrize('K,F,C', [(1, 1, 1), (3, 1, 1), (3, 3, 2), (8, 4, 4), (2, 1, 8)])
def test_class_split_shapes(cuda_lib, P, K, F, C):
    from pairhmm import _lib, api, synth
    rng = np.random.default_rng(P * 100 + K * F * C)
    p = synth.mixdom2_params(rng, K, F, C)
    if C > 1:
        p['classdist'][0, 0] = np.eye(C)[0]      # a group of one class only
    ts = rng.uniform(0.05, 2.0, P)
    pro = _lib.MixDom2Prologue(p)
    csubs = pro(ts)[4]
    cM = torch.tensor(rng.uniform(0, 2, (P, K * F, 21, 21)) * (rng.random((P, K * F, 21, 21)) < 0.6))
    cI, cD = (torch.tensor(rng.uniform(0, 2, (P, K * F, 21))) for _ in range(2))
    got = pro.class_counts(csubs, cM.cuda(), cI.cuda(), cD.cuda())
    want = api.class_split(p, cM, cI, cD, csubs=csubs.cpu())
    for k, w in want.items():
        d = (got[k].cpu() - w).abs().reshape(P, -1).amax(1)
        assert bool((d <= 1e-12 * w.abs().reshape(P, -1).amax(1)).all()), k
