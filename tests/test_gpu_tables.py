"""The lattice tables of phmm_estep_tables (wavefronts that leave value and exponent, tables_kernel after them) where the
generic stripes change: rows around the 32-row stripes, columns around the 8-column halo chunks, padded quads (5, 17 and
22 states), every table alone and together, wildcards, against the float64 oracle.  Bars of the float32 recursion as for
the reference's tables elsewhere: logs 1e-5 absolute where reachable, posteriors 1e-5, counts 1e-5 of the largest."""
import numpy as np
import pytest

from test_gpu_viterbi_stripes import model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('name', ['tkf', 'mixdom17', 'mixdom22'])
@pytest.mark.parametrize('shape', [(31, 7), (32, 8), (33, 9), (64, 25), (0, 5), (6, 0), (0, 0)])
def test_tables_match_oracle(cuda_lib, name, shape):
    from pairhmm import _lib, api, synth
    from oracle import dp, estep, models as om
    rng = np.random.default_rng(37)
    lt, st = model(name, rng)
    Q, pi, _ = synth.rand_Q_pi(rng)
    sub = om.transition_matrix(Q, 0.6)
    x, y = rng.integers(0, 21, shape[0]), rng.integers(0, 21, shape[1])
    EM, EI, ED = dp.group_tables_tkf(sub, pi)
    groups = np.zeros(len(st), int)
    emit = dp.log_emission_table(st, groups, x, y, EM, EI, ED)
    ll, post, n, F, B = dp.forward_backward(lt, st, emit)
    cM, cI, cD = estep.char_count_tables(post, st, groups, x, y, 1)
    plan = api.get_plan(st, groups, 1)
    batch = _lib.make_batch([x], [y], np.exp(lt)[None], EM[None], EI[None], ED[None])
    rows = np.isin(st, [0, 1, 2, 3])
    for want in [(1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1)]:
        out = _lib.estep_tables(plan, batch, *map(bool, want))
        assert abs(out['ll'][0].item() - ll) <= 1e-6 * max(abs(ll), 1.0)
        for key, ref, on in (('log_F', F, want[0]), ('log_B', B, want[1])):
            if on:
                got = out[key].cpu().numpy().reshape(ref.shape)[:, :, rows]
                live = ref[:, :, rows] > -1e29
                assert np.array_equal(got > -1e29, live), key
                assert np.abs(got - ref[:, :, rows])[live].max(initial=0.0) <= 1e-5, key
        if want[2]:
            np.testing.assert_allclose(out['post'].cpu().numpy().reshape(post.shape), post, atol=1e-5)
        for key, ref in (('n_trans', n), ('cnt_M', cM), ('cnt_I', cI), ('cnt_D', cD)):
            got = out[key][0].cpu().numpy()
            assert np.abs(got - ref).max() <= 1e-5 * max(ref.max(), 1e-3), key
