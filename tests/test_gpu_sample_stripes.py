"""The sampler's probability-space forward stripes (phmm_sample_paths) at stripe edges (32, 16, 8 rows), every lane shape,
and where they hand a pair to the log-space kernel (a table entry outside e^+-230, states far below their cell's
largest, a likelihood of zero), against the float64 oracle.  Log-likelihoods to 1e-12 relative (float64 on both sides,
sums of at most 64 positive terms a step); paths draw for draw."""
import numpy as np
import pytest

from test_gpu_viterbi_stripes import model

pytestmark = pytest.mark.gpu

CASES = [('tkf', [(31, 5), (32, 8), (33, 63), (64, 3), (0, 9), (7, 0), (0, 0)]),
         ('mixfrag2', [(15, 9), (16, 4), (17, 30)]),
         ('mixdom17', [(7, 16), (8, 15), (9, 1), (25, 20), (0, 5), (5, 0)]),
         ('mixdom22', [(7, 4), (8, 9), (17, 12)]),
         ('mixdom42', [(7, 8), (8, 7), (9, 9), (17, 3)])]


def check(lt, st, xs, ys, sub, pi, n=6, seed=5):
    from pairhmm import api
    from oracle import dp, sample
    ll, paths = api.sample_traceback_2d_batch(lt, st, xs, ys, sub, pi, n, seed=seed)
    EM, EI, ED = dp.group_tables_tkf(sub, pi)
    for b in range(len(xs)):
        emit = dp.log_emission_table(st, np.zeros(len(st), int), xs[b], ys[b], EM, EI, ED)
        want, wpaths = sample.sample_paths(lt, st, emit, n, seed=seed, pair=b)
        assert abs(ll[b] - want) <= 1e-12 * abs(want), b
        assert paths[b] == [[tuple(int(c) for c in v) for v in w] for w in wpaths], b


@pytest.mark.parametrize('name,shapes', CASES, ids=[c[0] for c in CASES])
def test_matches_oracle_at_stripe_edges(cuda_lib, name, shapes):
    from pairhmm import synth
    from oracle import models as om
    rng = np.random.default_rng(27)
    lt, st = model(name, rng)
    Q, pi, _ = synth.rand_Q_pi(rng)
    check(lt, st, [rng.integers(0, 20, a) for a, _ in shapes], [rng.integers(0, 20, b) for _, b in shapes],
          om.transition_matrix(Q, 0.6), pi)


@pytest.mark.parametrize('kind', ['tiny_transition', 'far_states', 'no_path'])
def test_pairs_outside_the_range_take_the_log_space_kernel(cuda_lib, kind):
    from pairhmm import synth
    from oracle import models as om
    rng = np.random.default_rng(28)
    lt, st = model('tkf', rng)
    Q, pi, _ = synth.rand_Q_pi(rng)
    lt = lt.copy()
    if kind == 'tiny_transition':
        lt[1, 3] = -500.0
    elif kind == 'far_states':   # deletions 2^-320 behind after two of them, each entry within range
        lt[:, 3] = np.where(lt[:, 3] > -1e29, -111.0, lt[:, 3])
    else:                        # no way to insert: pairs with Ly > Lx have none
        lt[:, 2] = -1e30
    shapes = [(40, 33), (5, 6), (12, 12)] if kind != 'no_path' else [(12, 9), (20, 20)]
    xs = [rng.integers(0, 20, a) for a, _ in shapes]
    ys = [rng.integers(0, 20, b) for _, b in shapes]
    check(lt, st, xs, ys, om.transition_matrix(Q, 0.6), pi)
    if kind == 'no_path':
        from pairhmm import api
        ll, _ = api.sample_traceback_2d_batch(lt, st, [xs[0][:3]], [ys[1]], om.transition_matrix(Q, 0.6), pi, 0)
        assert ll[0] <= -1e29
