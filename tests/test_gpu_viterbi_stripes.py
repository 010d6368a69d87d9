"""The Viterbi stripes (phmm_viterbi) at the sizes where they can go wrong: lengths around the stripe heights (64, 32,
16, 8 rows) and the four-column edge groups, every lane shape (4 to 64 slots), exact ties, impossible (-inf, NEG_INF)
transitions and envelopes, against the float64 oracle.  Both sides add the same float64 numbers in the same order, so
values agree to the oracle's own log tables (1e-12 relative) and paths are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model(name, rng):
    from pairhmm import synth
    from pairhmm import models as pm
    from oracle import models as om
    if name == 'tkf':
        return om.safe_log(om.tkf92_trans(0.03, 0.035, 0.6, 0.5)), np.array([0, 1, 2, 3, 4])
    if name == 'mixfrag2':
        return (om.safe_log(om.mixfrag_trans(0.03, 0.035, 0.6, [0.4, 0.7], [0.6, 0.4])), np.asarray(om.mixfrag_state_types(2)))
    K, F = {'mixdom17': (3, 1), 'mixdom22': (4, 1), 'mixdom42': (4, 2)}[name]
    p = synth.mixdom2_params(rng, K, F, 1)
    chi = om.build_nested_trans(p['main_ins'], p['main_del'], 0.6, p['dom_ins'], p['dom_del'], p['dom_weights'],
                                p['frag_weights'], p['ext_rates'])
    return om.safe_log(chi), pm.mixdom_state_types(K, F)


CASES = [('tkf', [(63, 5), (64, 8), (65, 63), (128, 3), (0, 9), (7, 0), (0, 0)]),
         ('mixfrag2', [(31, 9), (32, 4), (33, 30), (64, 1)]),
         ('mixdom17', [(15, 16), (16, 15), (17, 1), (33, 20), (0, 5), (5, 0)]),
         ('mixdom22', [(15, 4), (16, 9), (33, 12)]),
         ('mixdom42', [(7, 8), (8, 7), (9, 9), (17, 3)])]


@pytest.mark.parametrize('name,shapes', CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize('kind', ['plain', 'ties', 'minus_inf'])
def test_matches_oracle_at_stripe_edges(cuda_lib, name, shapes, kind):
    from pairhmm import api, synth
    from oracle import viterbi, models as om
    rng = np.random.default_rng(17)
    lt, st = model(name, rng)
    Q, pi, _ = synth.rand_Q_pi(rng)
    sub = om.transition_matrix(Q, 0.6)
    if kind == 'ties':   # every transition and residue alike: all paths of a length tie
        lt = np.where(lt > -1e29, -2.0, lt)
        pi, sub = np.full(20, 0.05), np.full((20, 20), 0.05)
    elif kind == 'minus_inf':
        lt = np.where(lt > -1e29, lt, -np.inf)
    xs = [rng.integers(0, 20, a) for a, _ in shapes]
    ys = [rng.integers(0, 20, b) for _, b in shapes]
    ll, paths = api.viterbi_2d_batch(lt, st, xs, ys, sub, pi)
    for b in range(len(shapes)):
        want, path = viterbi.viterbi_2d(lt, st, xs[b], ys[b], sub, pi)
        assert abs(ll[b] - want) <= 1e-12 * abs(want), b
        assert paths[b] == [tuple(v) for v in path], b


@pytest.mark.parametrize('name,shape', [('tkf', (70, 61)), ('mixdom17', (34, 30)), ('mixdom42', (18, 13))])
def test_envelope_across_stripes(cuda_lib, name, shape):
    from pairhmm import api, synth
    from oracle import beam, models as om
    rng = np.random.default_rng(18)
    lt, st = model(name, rng)
    Q, pi, _ = synth.rand_Q_pi(rng)
    sub = om.transition_matrix(Q, 0.6)
    x, y = rng.integers(0, 20, shape[0]), rng.integers(0, 20, shape[1])
    i, j = np.mgrid[0:shape[0] + 1, 0:shape[1] + 1]
    for width in (3, 9, 0):   # the last: an envelope no path fits in
        env = np.abs(j - i * shape[1] / shape[0]) <= width
        want, path = beam.beam_viterbi(lt, st, x, y, sub, pi, envelope=env)
        lp, got = api.beam_viterbi_2d(lt, st, x, y, sub, pi, envelope=env)
        assert abs(lp - want) <= 1e-12 * abs(want), width
        assert got == [tuple(int(c) for c in v) for v in path], width
