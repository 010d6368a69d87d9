"""The calls this library is used for, as measurable cases.

Each case is one call of the library as a user's program makes it: the
batched E-steps of EM and variational training (MixDom2 at 17, 42 and 162
states, TKF92), the differentiable log-likelihoods of gradient training, the
alignment-conditioned (1D) E-step and its gradient, the banded E-step, and
the decoders (Viterbi, sampled paths, posterior tables).  Inputs follow the
laws of the benchmark configurations: amino-acid sequences whose descendants
share about four fifths of their residues with the ancestor, insertion rates
U(0.01, 0.05), times LogUniform(0.05, 2), fragment extensions U(0.3, 0.9).
Lengths belong to a case (log-spaced over its range); sequences, times and
parameters come from the seed, as from one training iteration to the next.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (_ROOT, os.path.join(_ROOT, 'tkf-mixdom_gb300')):
    if _p not in sys.path:
        sys.path.insert(0, _p)

A = 20
S, M, I, D, E = 0, 1, 2, 3, 4
F64 = torch.float64


def listed():
    return [
        # one short pair under the 17-state model: a single E-step request, all latency
        {'name': 'mixdom17_estep_pair', 'kind': 'estep', 'K': 3, 'F': 1, 'C': 1, 'pairs': 1, 'lo': 45, 'hi': 46},
        # the held-out likelihood of a small validation set (64 pairs, lengths 50-150)
        {'name': 'tkf92_forward_64', 'kind': 'tkf92_forward', 'pairs': 64, 'lo': 50, 'hi': 150},
        # one minibatch of TKF92 variational training with its birth-death statistics
        {'name': 'tkf92_estep_512', 'kind': 'tkf92_estep', 'pairs': 512, 'lo': 50, 'hi': 400},
        # the benchmark's headline: a 17-state EM iteration over 200 pairs of 30-600 residues
        {'name': 'mixdom17_estep_200', 'kind': 'estep', 'K': 3, 'F': 1, 'C': 1, 'pairs': 200, 'lo': 30, 'hi': 600},
        # gradient training of the 42-state model (two fragment types, two site classes)
        {'name': 'mixdom42_grad_32', 'kind': 'grad', 'K': 4, 'F': 2, 'C': 2, 'pairs': 32, 'lo': 200, 'hi': 1500},
        # the 162-state model on a few long pairs, the largest state space of the benchmark
        {'name': 'mixdom162_estep_4', 'kind': 'estep', 'K': 8, 'F': 4, 'C': 4, 'pairs': 4, 'lo': 700, 'hi': 1100},
        # E-step in a band around guide alignments, posteriors in band layout
        {'name': 'tkf92_banded_64', 'kind': 'banded', 'pairs': 64, 'lo': 400, 'hi': 600, 'width': 36},
        # EM along given alignments (pair records of alignment databases)
        {'name': 'aligned17_estep_256', 'kind': 'aligned_estep', 'K': 3, 'F': 1, 'C': 1, 'pairs': 256, 'lo': 40,
         'hi': 500},
        # gradient training along given alignments, 42 states
        {'name': 'aligned42_grad_64', 'kind': 'aligned_grad', 'K': 4, 'F': 2, 'C': 2, 'pairs': 64, 'lo': 60,
         'hi': 400},
        # most probable alignments of a family's pairs under the 17-state model
        {'name': 'mixdom17_viterbi_24', 'kind': 'viterbi', 'K': 3, 'F': 1, 'C': 1, 'pairs': 24, 'lo': 80, 'hi': 400},
        # alignments sampled from the posterior, as an alignment sampler proposes them
        {'name': 'tkf92_sample_16', 'kind': 'sample', 'pairs': 16, 'lo': 60, 'hi': 300, 'samples': 32},
        # one pair with its whole posterior table, as a caller looks at a single alignment
        {'name': 'tkf92_posteriors_pair', 'kind': 'posteriors', 'pairs': 1, 'lo': 150, 'hi': 151},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind of call, a model of that kind, a batch size and a range of lengths."""
    kind = rng.choice(['estep', 'estep', 'tkf92_forward', 'tkf92_estep', 'grad', 'banded', 'aligned_estep',
                       'aligned_grad', 'viterbi', 'sample', 'posteriors'])
    c = {'kind': kind}
    if kind in ('estep', 'grad'):
        c['K'], c['F'], c['C'] = rng.choice([(3, 1, 1), (3, 1, 1), (4, 2, 2), (8, 4, 4)] if kind == 'estep'
                                            else [(3, 1, 1), (4, 2, 2)])
        n = 2 + 5 * c['K'] * c['F']
        c['pairs'] = _log_uniform(rng, 1, {17: 200, 42: 32, 162: 4}[n])
        top = {17: 600, 42: 1400, 162: 1000}[n]
    elif kind in ('aligned_estep', 'aligned_grad'):
        c['K'], c['F'], c['C'] = rng.choice([(3, 1, 1), (4, 2, 2)])
        c['pairs'] = _log_uniform(rng, 4, 256 if kind == 'aligned_estep' else 64)
        top = 500
    elif kind == 'viterbi':
        c['K'], c['F'], c['C'] = rng.choice([(0, 0, 0), (3, 1, 1), (4, 2, 2)])
        c['pairs'] = _log_uniform(rng, 1, 24)
        top = 400 if c['K'] < 4 else 200
    else:
        c['pairs'] = 1 if kind == 'posteriors' else _log_uniform(
            rng, 4, {'tkf92_forward': 512, 'tkf92_estep': 512, 'banded': 64, 'sample': 16}[kind])
        top = {'tkf92_forward': 400, 'tkf92_estep': 400, 'banded': 600, 'sample': 300, 'posteriors': 300}[kind]
    c['lo'] = _log_uniform(rng, 20, top // 2)
    c['hi'] = max(c['lo'] + 1, _log_uniform(rng, c['lo'] + 1, top))
    if kind == 'banded':
        c['width'] = rng.randint(8, 48)
    if kind == 'sample':
        c['samples'] = _log_uniform(rng, 1, 64)
    return c


# ---------------------------------------------------------------- inputs
def _lengths(case):
    """Ancestor and descendant lengths of the case's pairs (the same for every seed)."""
    n = case['pairs']
    q = np.random.RandomState(7).permutation(n)
    lx = np.rint(case['lo'] * (case['hi'] / case['lo']) ** ((q + 0.5) / n)).astype(int)
    golden = (np.arange(n) * 0.6180339887498949 + 0.3) % 1.0
    return lx, np.maximum(1, np.rint(lx * (0.85 + 0.3 * golden)).astype(int))


def _reversible(rng):
    """(exchangeabilities, frequencies) of one site class, one expected substitution per unit time."""
    pi = rng.dirichlet(np.ones(A))
    ex = np.triu(rng.lognormal(0.0, 1.0, (A, A)), 1)
    ex = ex + ex.T
    return ex / (pi @ ex @ pi), pi


def _rate_matrix(ex, pi):
    q = ex * pi[None, :]
    np.fill_diagonal(q, 0.0)
    np.fill_diagonal(q, -q.sum(axis=1))
    return q


def _mixdom2_params(rng, K, F, C):
    cls = [_reversible(rng) for _ in range(C)]
    lam, dom = rng.uniform(0.01, 0.05), rng.uniform(0.01, 0.05, K)
    return {'main_ins': lam, 'main_del': lam * rng.uniform(1.05, 1.5),
            'dom_ins': dom, 'dom_del': dom * rng.uniform(1.05, 1.5, K), 'dom_weights': rng.dirichlet(np.ones(K)),
            'frag_weights': rng.dirichlet(np.ones(F), K), 'ext_rates': rng.uniform(0.3, 0.9, (K, F)),
            'class_pis': np.stack([c[1] for c in cls]), 'class_S_exch': np.stack([c[0] for c in cls]),
            'classdist': rng.dirichlet(np.ones(C), (K, F))}


def _tkf_params(rng):
    ex, pi = _reversible(rng)
    lam = rng.uniform(0.01, 0.05)
    return {'lam': lam, 'mu': lam * rng.uniform(1.05, 1.5), 'ext': rng.uniform(0.3, 0.9),
            'Q': _rate_matrix(ex, pi), 'pi': pi}


def _descendant(rng, x, ly):
    """A homologous sequence of ly residues: about nine tenths of the shorter one aligned, three in four of those
    unchanged, the rest inserted anywhere."""
    keep = max(1, int(0.9 * min(len(x), ly)))
    kept = x[np.sort(rng.permutation(len(x))[:keep])]
    kept = np.where(rng.random(keep) < 0.25, rng.integers(0, A, keep), kept)
    y = rng.integers(0, A, ly)
    y[np.sort(rng.permutation(ly)[:keep])] = kept
    return y


def _alignment(rng, n):
    """Column types (1 match, 2 insert, 3 delete) in runs, and the characters of an n-column alignment."""
    runs = rng.geometric(0.2, n)
    types = rng.choice([1, 1, 1, 1, 2, 3], n)
    cols = np.repeat(types, runs)[:n].astype(np.uint8)
    anc = rng.integers(0, A, n)
    desc = np.where(rng.random(n) < 0.7, anc, rng.integers(0, A, n))
    anc, desc = np.where(cols == 2, A, anc), np.where(cols == 3, A, desc)
    return cols, anc.astype(np.uint8), desc.astype(np.uint8)


def _inputs(case, seed):
    """Host inputs of a case: parameters, times, sequences or alignments."""
    rng = np.random.default_rng([seed, 20, case['pairs']])
    mixdom = case.get('K', 0) > 0
    p = _mixdom2_params(rng, case['K'], case['F'], case['C']) if mixdom else _tkf_params(rng)
    lx, ly = _lengths(case)
    s = {'p': p, 'ts': np.exp(rng.uniform(math.log(0.05), math.log(2.0), case['pairs']))}
    if case['kind'].startswith('aligned'):
        s['cols'], s['ancs'], s['descs'] = (list(v) for v in zip(*(_alignment(rng, int(n)) for n in lx)))
    else:
        s['xs'] = [rng.integers(0, A, int(n)) for n in lx]
        s['ys'] = [_descendant(rng, x, int(n)) for x, n in zip(s['xs'], ly)]
    if case['kind'] == 'banded':   # guides near the diagonal
        s['centers'] = [np.rint(np.arange(a + 1) * (b / a)).astype(np.int32) for a, b in zip(lx, ly)]
    return s


_GRAD_ARGS = ('main_ins', 'main_del', 't', 'dom_ins', 'dom_del', 'dom_weights', 'frag_weights', 'ext_rates',
              'class_pis', 'class_S_exch', 'classdist')


def _log(v):
    v = np.asarray(v, np.float64)
    return np.where(v > 0, np.log(np.maximum(v, 1e-300)), -1e30)


def prepare(case, seed):
    from pairhmm import _lib, api
    s = _inputs(case, seed)
    p, kind = s['p'], case['kind']
    s['kind'], s['case'] = kind, case
    if kind.startswith('tkf92_'):   # padded arrays, as the minibatch loader makes them
        pad = lambda seqs: np.stack([np.pad(v, (0, max(map(len, seqs)) - len(v))) for v in seqs])
        s['x_pad'], s['y_pad'] = pad(s['xs']), pad(s['ys'])
        s['lx'], s['ly'] = np.array([len(x) for x in s['xs']]), np.array([len(y) for y in s['ys']])
    elif kind in ('grad', 'aligned_grad'):   # the training program's leaf tensors
        vals = dict(p, t=s['ts'])
        s['leaves'] = {k: torch.tensor(vals[k], dtype=F64, device='cuda', requires_grad=True) for k in _GRAD_ARGS}
    elif kind == 'banded':   # a plan and a device batch with its band masks
        chi, EM, EI, ED = (v.cpu() for v in _tkf_model(p, s['ts'], 'cpu'))
        st = np.array([S, M, I, D, E])
        s['plan'] = api.get_plan(st, np.zeros(5, np.int32), 1)
        masks = [np.where(np.abs(np.arange(len(y) + 1)[None, :] - c[:, None]) <= case['width'], 7, 0).astype(np.uint8)
                 for y, c in zip(s['ys'], s['centers'])]
        s['batch'] = _lib.make_batch(s['xs'], s['ys'], chi, EM, EI, ED, device='cuda', cell_masks=masks)
    elif kind in ('viterbi', 'sample'):   # log tables on the device
        st, gr = _states(case)
        tabs = _model(case, p, s['ts'], 'cpu')
        s['st'], s['gr'], s['G'] = st, gr, int(gr.max()) + 1
        s['logs'] = [torch.from_numpy(_log(v.numpy())).cuda() for v in tabs]
    elif kind == 'posteriors':
        s['log_chi'] = _log(_tkf_model(p, s['ts'], 'cpu')[0][0].numpy())
        s['sub'] = torch.linalg.matrix_exp(torch.from_numpy(p['Q'] * s['ts'][0])).numpy()
    return s


def _paths(s, paths):
    """The paths in one padded array, as a caller keeps those of a batch, and their lengths."""
    most = max(len(x) + len(y) + 1 for x, y in zip(s['xs'], s['ys']))
    out = np.zeros((len(paths), most, 3), np.int32)
    for row, v in zip(out, paths):
        row[:len(v)] = v
    return {'paths': out, 'lengths': np.array([len(v) for v in paths])}


def run(s):
    from pairhmm import _lib, api
    kind, p = s['kind'], s['p']
    if kind == 'estep':
        return api.estep_batch_mixdom2(p, s['xs'], s['ys'], s['ts'])
    if kind == 'tkf92_forward':
        return api.estep_batch_tkf92_forward_only(s['x_pad'], s['y_pad'], s['ts'], s['lx'], s['ly'], p['lam'],
                                                  p['mu'], p['ext'], p['Q'], p['pi'])
    if kind == 'tkf92_estep':
        return api.estep_batch_tkf92(s['x_pad'], s['y_pad'], s['ts'], s['lx'], s['ly'], p['lam'], p['mu'], p['ext'],
                                     p['Q'], p['pi'])
    if kind == 'banded':
        out = dict(_lib.estep_band(s['plan'], s['batch'], s['centers'], s['case']['width']))
        out.pop('_centers')
        return out
    if kind == 'aligned_estep':
        return api.estep_1d_mixdom2(p, s['cols'], s['ancs'], s['descs'], s['ts'])
    if kind in ('grad', 'aligned_grad'):
        q = s['leaves']
        for v in q.values():
            v.grad = None
        if kind == 'grad':
            ll = api.mixdom2_log_prob(*(q[k] for k in _GRAD_ARGS), s['xs'], s['ys'])
        else:
            ll = api.mixdom2_constrained_log_prob(
                *(q[k] for k in _GRAD_ARGS[:8]), q['class_S_exch'], q['class_pis'], q['classdist'], s['cols'],
                s['ancs'], s['descs'])
        (-ll.sum()).backward()
        return {'log_p': ll.detach(), **{k: v.grad for k, v in q.items()}}
    if kind == 'viterbi':
        ll, paths = _lib.viterbi(s['st'], s['gr'], s['G'], s['xs'], s['ys'], *s['logs'])
        return {'log_p': ll, **_paths(s, paths)}
    if kind == 'sample':
        ll, paths = _lib.sample_paths(s['st'], s['gr'], s['G'], s['xs'], s['ys'], *s['logs'], s['case']['samples'],
                                      11)
        return {'log_p': ll, **_paths(s, [v for per_pair in paths for v in per_pair])}
    ll, post, n = api.forward_backward_2d(s['log_chi'], np.array([S, M, I, D, E]), s['xs'][0], s['ys'][0], s['sub'],
                                          p['pi'])
    return {'log_p': ll, 'posteriors': post, 'n_trans': n}


def work(case):
    """Inputs read once and outputs written once; the multiply-adds of each recursion through the factors the
    transitions are made of (main type sums plus same-domain blocks), and one per state pair for the counts."""
    lx, ly = _lengths(case)
    K, F, C, P = case.get('K', 0), case.get('F', 1), case.get('C', 1), case['pairs']
    body = 5 * K * F if K else 3
    n = 2 + body
    G = max(1, K * F)
    step = 6 * body + 11 * K * F * F if K else 9        # multiply-adds of one cell and pass
    cells = float(((lx + 1) * (ly + 1)).sum())
    params = 8.0 * (A * A * C + (n * n if K else 3))
    seqs = float((lx + ly).sum())
    counts = 8.0 * P * (n * n + G * (441 + 42))
    kind = case['kind']
    if kind == 'banded':
        cells = float(sum((a + 1) * min(b + 1, 2 * case['width'] + 1) for a, b in zip(lx, ly)))
        return {'bytes': seqs + cells + counts + 8.0 * cells * n, 'flops': cells * (4 * step + 2 * body * body)}
    if kind.startswith('aligned'):
        cols = float(lx.sum())
        third = body / 3.0                                # states of a column's own type
        return {'bytes': 3 * cols + params + counts, 'flops': cols * 6 * third * third + 2e4 * P}
    if kind == 'tkf92_forward':
        return {'bytes': seqs + params + 8.0 * P, 'flops': cells * 2 * step}
    if kind == 'viterbi':                                 # an addition and a comparison per transition
        return {'bytes': seqs + 8.0 * P * (n * n + G * 483) + 12 * seqs, 'flops': cells * 2 * body * body}
    if kind == 'sample':
        return {'bytes': seqs + 8.0 * P * (n * n + G * 483) + 12 * seqs * case['samples'],
                'flops': cells * 2 * step + seqs * case['samples'] * 3 * body}
    if kind == 'posteriors':
        return {'bytes': seqs + 8.0 * cells * n, 'flops': cells * (4 * step + 2 * body * body)}
    return {'bytes': seqs + params + counts, 'flops': cells * (4 * step + 2 * body * body)}


# ---------------------------------------------------------------- the same in 64 bits
def _tkf91(lam, mu, t):
    lam, mu, t = torch.broadcast_tensors(lam, mu, t)
    a, e = torch.exp(-mu * t), torch.exp(-lam * t)
    b = lam * (e - a) / (mu * e - lam * a)
    g = 1 - mu * b / (lam * (1 - a))
    k = lam / mu
    z = torch.zeros_like(a)
    row = lambda h: torch.stack([z, (1 - h) * k * a, h, (1 - h) * k * (1 - a), (1 - h) * (1 - k)], -1)
    return torch.stack([row(b), row(b), row(b), row(g), torch.stack([z] * 5, -1)], -2)


def _pad1(v, dims):
    for d in dims:
        v = torch.cat([v, torch.ones_like(v.narrow(d, 0, 1))], d)
    return v


def _tkf_model(p, ts, dev, floor=True):
    """TKF92 transitions [P,5,5] and character tables, float64."""
    f = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=dev)
    t = f(ts)
    t91 = _tkf91(f(p['lam']), f(p['mu']), t)
    emit = torch.tensor([0., 1., 1., 1., 0.], dtype=F64, device=dev)
    chi = t91 * (1 - p['ext'] * emit)[:, None] + p['ext'] * torch.diag(emit)
    if floor:
        chi = chi.clamp_min(1e-30)
    pi = _pad1(f(p['pi']) + 1e-30, [0]).expand(len(ts), 21)
    sub = _pad1(torch.linalg.matrix_exp(t[:, None, None] * f(p['Q'])) + 1e-30, [1, 2])
    return chi, (pi[:, :, None] * sub)[:, None], pi[:, None], pi[:, None]


def _mixdom2_model(q):
    """Collapsed MixDom2 transitions [P,N,N] and character tables from float64 tensors, differentiable."""
    t, w, fw, ext = q['t'], q['dom_weights'], q['frag_weights'], q['ext_rates']
    (K, F), P, dev = fw.shape, t.numel(), t.device
    top = _tkf91(q['main_ins'], q['main_del'], t)                                   # P,5,5
    dom = _tkf91(q['dom_ins'], q['dom_del'], t[:, None])                            # P,K,5,5
    kap = q['dom_ins'] / q['dom_del']
    ends = dom[:, :, S, E]                                                          # an empty domain, with time
    mid = [M, I, D]
    # a chain over top-level links that passes through empty domains (M, I, D links of domain k)
    empty = torch.stack([ends, (1 - kap).expand(P, K), (1 - kap).expand(P, K)], -1)  # P,K,3
    full = torch.stack([1 - ends, kap.expand(P, K), kap.expand(P, K)], -1)
    rows = top[:, [M, M, D]]                       # an empty M link leaves as M, I as M, D as D
    enter = (top[:, :, mid][:, :, None, :] * w[:, None]).reshape(P, 5, 3 * K)
    hop = (empty[..., None, None] * rows[:, None, :, None, mid] * w[:, None]).reshape(P, 3 * K, 3 * K)
    leave = torch.zeros(P, K, 3, 5, dtype=F64, device=dev)
    leave = leave + torch.diag_embed(full)[..., [0, 0, 1, 2, 2]] * torch.tensor([0., 1., 1., 1., 0.], device=dev)
    tail = empty * rows[:, None, :, E]
    leave = leave + tail[..., None] * torch.tensor([0., 0., 0., 0., 1.], device=dev)
    closure = torch.linalg.inv(torch.eye(3 * K, dtype=F64, device=dev) - hop).reshape(P, 3 * K, K, 3)
    T = torch.einsum('pui,pike,pkev->pkuv', enter, closure, leave)                  # P,K,5,5
    T_all = T.sum(1) + top * torch.tensor([0., 0., 0., 0., 1.], device=dev)
    # body states (domain, pair of link types, fragment): MM MI MD II DD
    U, X, is_m = [M, M, M, I, D], [M, I, D, I, D], torch.tensor([1., 1., 1., 0., 0.], device=dev)
    entry = is_m * dom[:, :, S, X] / (1 - ends)[..., None] + (1 - is_m)
    out = is_m * dom[..., E][..., X] + (1 - is_m) * (1 - kap)[:, None]
    stop = 1 - ext                                                                  # K,F
    ex = (stop[:, None, :] * out[..., None]).reshape(P, -1)
    en = (fw[:, None, :] * entry[..., None]).reshape(P, -1)
    nb, bs = 5 * K * F, 5 * F
    d_of, v_of = torch.arange(nb) // bs, (torch.arange(nb) % bs) // F
    u_of = torch.tensor(U)[v_of]
    body = ex[:, :, None] * T[:, d_of[None, :], u_of[:, None], u_of[None, :]] * en[:, None, :]
    links = torch.zeros(P, K, 5, 5, dtype=F64, device=dev)
    links[:, :, :3, :3] = dom[:, :, 1:4, 1:4]
    links[:, :, 3, 3] = links[:, :, 4, 4] = kap
    intra = torch.einsum('kf,pkuv,kg->pkufvg', stop, links, fw)
    eye5, eyeF = torch.eye(5, dtype=F64, device=dev), torch.eye(F, dtype=F64, device=dev)
    intra = (intra + torch.einsum('kf,uv,fg->kufvg', ext, eye5, eyeF)).reshape(P, K, bs, bs)
    body = body + torch.stack([torch.block_diag(*blk) for blk in intra])
    n = 2 + nb
    chi = torch.zeros(P, n, n, dtype=F64, device=dev)
    chi[:, 0, 1] = T_all[:, S, E]
    chi[:, 0, 2:] = T[:, d_of, S, u_of] * en
    chi[:, 2:, 1] = ex * T_all[:, u_of, E]
    chi[:, 2:, 2:] = body
    Q = q['class_S_exch'] * q['class_pis'][:, None, :]
    Q = Q - torch.diag_embed(torch.diagonal(Q, dim1=-2, dim2=-1))
    Q = Q - torch.diag_embed(Q.sum(-1))
    sub = torch.linalg.matrix_exp(t[:, None, None, None] * Q)                       # P,C,A,A
    cd = q['classdist'].reshape(K * F, -1)
    pi = _pad1(q['class_pis'], [1])
    EM = torch.einsum('gc,ca,pcab->pgab', cd, pi, _pad1(sub, [2, 3]))
    EI = (cd @ pi).expand(P, K * F, 21)
    return chi, EM, EI, EI, sub


def _states(case):
    K, F = case.get('K', 0), case.get('F', 0)
    if not K:
        return np.array([S, M, I, D, E]), np.zeros(5, np.int32)
    b = np.arange(5 * K * F)
    st = np.concatenate([[S, E], np.array([M, I, D, I, D])[(b % (5 * F)) // F]])
    return st.astype(np.int8), np.concatenate([[0, 0], (b // (5 * F)) * F + b % F]).astype(np.int32)


def _tensors(p, ts, dev):
    vals = dict(p, t=ts)
    return {k: torch.tensor(vals[k], dtype=F64, device=dev) for k in _GRAD_ARGS}


def _model(case, p, ts, dev):
    return _mixdom2_model(_tensors(p, ts, dev))[:4] if case.get('K', 0) else _tkf_model(p, ts, dev)


def _pad(seqs, value=0):
    return torch.from_numpy(np.stack([np.pad(np.asarray(v, np.int64), (0, max(map(len, seqs)) - len(v)),
                                             constant_values=value) for v in seqs]))


def _lattice(st, gr, tabs, xs, ys, dev, want='counts', band=None, viterbi=False):
    """Forward, backward, posteriors and counts of a batch on whole anti-diagonals, float64, each diagonal scaled
    by its largest value.  band: (centres, half width).  want: 'll', 'counts' or 'posteriors'."""
    chi, EM, EI, ED = (v.to(dev) for v in tabs)
    if viterbi:
        chi = torch.log(chi)
    P, G, n = len(xs), EM.shape[1], len(st)
    X, Y = _pad(xs).to(dev), _pad(ys).to(dev)
    Lx, Ly = (torch.tensor([len(v) for v in q], device=dev) for q in (xs, ys))
    R = X.shape[1] + 1                               # rows of a diagonal
    rows = torch.arange(R, device=dev)
    st_t, gr_t = torch.as_tensor(np.asarray(st, np.int64), device=dev), torch.as_tensor(np.asarray(gr, np.int64), device=dev)
    kind = [(st_t == ty).nonzero()[:, 0] for ty in (M, I, D)]
    e_col = int(np.argmax(np.asarray(st) == E))
    pr = torch.arange(P, device=dev)[:, None]
    xi = torch.cat([torch.zeros(P, 1, dtype=torch.long, device=dev), X], 1)[:, :R]
    cent = None if band is None else _pad(band[0], 1 << 20).to(dev)
    last = int((Lx + Ly).max())

    def cells(d):
        """Valid cells, their emissions [P,R,n] and residues on diagonal d."""
        j = d - rows[None, :]
        ok = (rows[None, :] <= Lx[:, None]) & (j >= 0) & (j <= Ly[:, None])
        if cent is not None:
            ok = ok & ((j - cent).abs() <= band[1])
        yj = torch.gather(Y, 1, (j - 1).clamp(0, Y.shape[1] - 1).expand(P, R))
        e = torch.zeros(P, R, n, dtype=F64, device=dev)
        i1, j1 = (rows >= 1)[None, :], j >= 1
        for ks, tab, on in ((kind[0], EM[pr, :, xi, yj], ok & i1 & j1), (kind[1], EI[pr, :, yj], ok & j1),
                            (kind[2], ED[pr, :, xi], ok & i1)):
            e[:, :, ks] = tab[:, :, gr_t[ks]] * on[..., None]
        return ok, e, yj

    def step(f, k, c):
        if not viterbi:
            return f @ c[:, :, k]
        return torch.stack([(f + c[:, None, :, int(q)]).amax(-1) for q in k], -1)

    zero = -math.inf if viterbi else 0.0
    blank = torch.full((P, R, n), zero, dtype=F64, device=dev)
    down = lambda v: torch.cat([blank[:, :1], v[:, :-1]], 1)
    f = blank.clone()
    f[:, 0, 0] = 0.0 if viterbi else 1.0
    fs, sc = [f], [torch.zeros(P, dtype=F64, device=dev)]
    end = [None] * P
    done = (Lx + Ly).tolist()
    for d in range(last + 1):
        if d:
            _, e, _ = cells(d)
            two = fs[-2] if d > 1 else blank
            two_s = sc[-2] if d > 1 else sc[-1]
            f = torch.full((P, R, n), zero, dtype=F64, device=dev)
            gap = two_s - sc[-1]
            m = step(down(two), kind[0], chi)
            f[:, :, kind[0]] = m + gap[:, None, None] if viterbi else m * torch.exp(gap)[:, None, None]
            f[:, :, kind[1]] = step(fs[-1], kind[1], chi)
            f[:, :, kind[2]] = step(down(fs[-1]), kind[2], chi)
            f = f + torch.log(e) if viterbi else f * e
            top = f.amax((1, 2))
            if viterbi:
                top = torch.where(torch.isfinite(top), top, torch.zeros_like(top))
                f, s = f - top[:, None, None], sc[-1] + top
            else:
                top = torch.where(top > 0, top, torch.ones_like(top))
                f, s = f / top[:, None, None], sc[-1] + torch.log(top)
            fs.append(f)
            sc.append(s)
            if want == 'll':
                fs[:-2] = []
                sc[:-2] = []
        for p in range(P):
            if done[p] == d:
                v, c = fs[-1][p, int(Lx[p])], chi[p, :, e_col]
                end[p] = (v + c).max() + sc[-1][p] if viterbi else torch.log((v * c).sum()) + sc[-1][p]
    ll = torch.stack(end)
    if want == 'll':
        return {'log_p': ll}
    N = torch.zeros(P, n, n, dtype=F64, device=dev)
    cM, cI, cD = (torch.zeros(P * G * k, dtype=F64, device=dev) for k in (441, 21, 21))
    post = None
    if want == 'posteriors':
        post = torch.zeros(P, R, int(Ly.max()) + 1, n, dtype=F64, device=dev)
    wb = [blank, blank]                               # e b on diagonals d+1 and d+2, with their scales
    ws = [torch.zeros(P, dtype=F64, device=dev)] * 2
    up = lambda v: torch.cat([v[:, 1:], blank[:, :1]], 1)
    for d in range(last, -1, -1):
        ok, e, yj = cells(d)
        w = torch.zeros(P, R, n, dtype=F64, device=dev)
        ref = torch.maximum(ws[0], ws[1])
        w[:, :, kind[0]] = up(wb[1])[:, :, kind[0]] * torch.exp(ws[1] - ref)[:, None, None]
        w[:, :, kind[1]] = wb[0][:, :, kind[1]] * torch.exp(ws[0] - ref)[:, None, None]
        w[:, :, kind[2]] = up(wb[0])[:, :, kind[2]] * torch.exp(ws[0] - ref)[:, None, None]
        here = (Lx + Ly == d).nonzero()[:, 0]
        for p in here.tolist():                       # the terminal cell steps to End
            w[p] = 0
            w[p, int(Lx[p]), e_col] = 1.0
            ref = ref.clone()
            ref[p] = 0.0
        live = (Lx + Ly >= d).to(F64)
        g = torch.exp(torch.where(live > 0, sc[d] + ref - ll, torch.zeros_like(ll))) * live
        N += (fs[d].transpose(1, 2) @ w) * g[:, None, None]
        b = w @ chi.transpose(1, 2)
        ga = fs[d] * b * g[:, None, None]
        if post is not None:
            i, p = rows[(d - rows >= 0) & (d - rows < post.shape[2])], slice(None)
            post[p, i, d - i] = ga[p, i]
        if d:
            for ks, acc, width, code in ((kind[0], cM, 441, xi * 21 + yj), (kind[1], cI, 21, yj), (kind[2], cD, 21, xi)):
                acc.index_add_(0, ((pr[..., None] * G + gr_t[ks]) * width + code[..., None]).reshape(-1),
                               ga[:, :, ks].reshape(-1))
        b = b * e
        top = b.amax((1, 2))
        top = torch.where(top > 0, top, torch.ones_like(top))
        wb, ws = [b / top[:, None, None], wb[0]], [ref + torch.log(top), ws[0]]
    return {'log_p': ll, 'n_trans': N * chi, 'cnt_M': cM.view(P, G, 21, 21), 'cnt_I': cI.view(P, G, 21),
            'cnt_D': cD.view(P, G, 21), 'posteriors': post}


def _chunks(s, n, per=12e9):
    """The batch's pairs in groups of like lengths whose forward diagonals take at most `per` bytes."""
    size = [len(x) + len(y) for x, y in zip(s['xs'], s['ys'])]
    group, out = [], []
    for p in np.argsort(size, kind='stable'):
        if group and 8.0 * n * size[p] * (len(group) + 1) * (1 + max(len(s['xs'][q]) for q in group + [p])) > per:
            out.append(group)
            group = []
        group.append(int(p))
    return out + [group]


def _batched(case, s, tabs, dev, **kw):
    st, gr = _states(case)
    got = {}
    for grp in _chunks(s, len(st)):
        r = _lattice(st, gr, [v[grp] for v in tabs], [s['xs'][p] for p in grp], [s['ys'][p] for p in grp], dev, **kw)
        for k, v in r.items():
            if v is not None:
                got.setdefault(k, [None] * len(s['xs']))
                for a, p in enumerate(grp):
                    got[k][p] = v[a]
    return {k: torch.stack(v) for k, v in got.items()}


def _class_counts(q, sub, cM, cI, cD):
    """Counts split over the site classes by each class's posterior given the residues."""
    K, F, C = q['classdist'].shape
    cd = q['classdist'].reshape(K * F, C)
    jM = cd[:, :, None, None] * (q['class_pis'][:, :, None] * sub)[:, None]            # P,G,C,A,A
    jI = cd[:, :, None] * q['class_pis']
    wM = cM[:, :, None, :A, :A] * jM / jM.sum(2, keepdim=True)
    share = jI / jI.sum(1, keepdim=True)
    wI, wD = cI[:, :, None, :A] * share, cD[:, :, None, :A] * share
    return {'class_match_counts': wM.sum(1), 'class_insert_counts': wI.sum(1), 'class_delete_counts': wD.sum(1),
            'classdist_counts': (wM.sum((-2, -1)) + wI.sum(-1) + wD.sum(-1)).view(-1, K, F, C)}


def _dwell(q, sub, t, n):
    """Expected dwell times and substitutions of each class from its match counts (eigendecomposition)."""
    W, U = [], []
    for c in range(sub.shape[1]):
        pi = q['class_pis'][c]
        Q = q['class_S_exch'][c] * pi
        Q = Q - torch.diag(Q.diagonal())
        Q = Q - torch.diag(Q.sum(1))
        r = pi.sqrt()
        sym = Q * r[:, None] / r
        lam, V = torch.linalg.eigh((sym + sym.T) / 2)
        ex = torch.exp(lam * t[:, None])
        diff = lam[:, None] - lam
        same = diff.abs() < 1e-10
        J = torch.where(same, t[:, None, None] * ex[:, :, None],
                        (ex[:, :, None] - ex[:, None, :]) / torch.where(same, torch.ones_like(diff), diff))
        L, Rt = V / r[:, None], V * r[:, None]        # P(t) = L e^(lam t) Rt^T
        inner = torch.einsum('ak,pab,bl->pkl', L, n[:, c] / sub[:, c], Rt) * J
        full = torch.einsum('ik,pkl,jl->pij', Rt, inner, L)
        W.append(full.diagonal(dim1=1, dim2=2))
        u = Q * full
        U.append(u - torch.diag_embed(u.diagonal(dim1=1, dim2=2)))
    return {'class_W': torch.stack(W, 1), 'class_U': torch.stack(U, 1)}


def _birth_death(n, p, ts, dev):
    """Fragment-resolved counts of TKF92 and the birth-death statistics from the scores of the link likelihood."""
    t = torch.as_tensor(ts, device=dev)
    lam = torch.full_like(t, p['lam']).requires_grad_()
    mu = torch.full_like(t, p['mu']).requires_grad_()
    chi = _tkf_model(p, ts, dev, floor=False)[0]
    dg = chi.diagonal(dim1=1, dim2=2)[:, 1:4]
    loops = n.diagonal(dim1=1, dim2=2)[:, 1:4]
    kept = (p['ext'] / dg).clamp(0, 1) * loops
    res = n - torch.nn.functional.pad(torch.diag_embed(kept), (1, 1, 1, 1))
    lk = torch.log(_tkf91(lam, mu, t).clamp_min(1e-300))
    # link likelihood without its kappa factors: divide each entry by (lam/mu) or (1 - lam/mu)
    k = torch.log(lam / mu), torch.log(1 - lam / mu)
    lk = torch.stack([lk[:, :, M] - k[0][:, None], lk[:, :, I], lk[:, :, D] - k[0][:, None], lk[:, :, E] - k[1][:, None]], -1)
    cnt = res[:, :4, 1:]
    lp = (cnt * lk[:, :4]).sum()
    dl, dm = torch.autograd.grad(lp, (lam, mu))
    ls, ms = p['lam'] * dl, p['mu'] * dm
    cons = res[:, :, I].sum(1) - res[:, :, D].sum(1)
    s_ = (cons + ms - ls - p['lam'] * t) / (p['lam'] - p['mu'])
    return {'B': (ls + p['lam'] * s_ + p['lam'] * t).clamp_min(0), 'D': (ms + p['mu'] * s_).clamp_min(0),
            'S': s_.clamp_min(0), 'L': res[:, :4][:, :, [M, D]].sum((1, 2)), 'M': res[:, :4, E].sum(1), 'T': t,
            'ext_count': kept.sum(1), 'notext_count': res[:, 1:4].sum((1, 2))}


def _along(case, s, tabs, dev):
    """Forward-backward along given alignments, float64: log-likelihood, transition and character counts."""
    chi, EM, EI, ED = (v.to(dev) for v in tabs)
    st, gr = _states(case)
    st_t, gr_t = torch.as_tensor(st.astype(np.int64), device=dev), torch.as_tensor(gr.astype(np.int64), device=dev)
    P, G, n = len(s['cols']), EM.shape[1], len(st)
    col, anc, des = (_pad(s[k]).to(dev) for k in ('cols', 'ancs', 'descs'))
    L = torch.tensor([len(c) for c in s['cols']], device=dev)
    e_col, top = int(np.argmax(st == E)), col.shape[1]
    pr = torch.arange(P, device=dev)
    em = torch.zeros(top, P, n, dtype=F64, device=dev)
    for c in range(top):
        for ty, tab in ((M, EM[pr, :, anc[:, c], des[:, c]]), (I, EI[pr, :, des[:, c]]), (D, ED[pr, :, anc[:, c]])):
            ks = (st_t == ty).nonzero()[:, 0]
            em[c][:, ks] = tab[:, gr_t[ks]] * (col[:, c] == ty)[:, None]
    a = torch.zeros(P, n, dtype=F64, device=dev)
    a[:, 0] = 1.0
    al, sc, s0 = [a], [torch.zeros(P, dtype=F64, device=dev)], None
    for c in range(top):
        v = torch.einsum('ps,psk->pk', al[-1], chi) * em[c]
        live = (c < L)[:, None]
        v = torch.where(live, v, al[-1])
        m = torch.where(live[:, 0], v.sum(1), torch.ones_like(v[:, 0]))
        al.append(v / m[:, None])
        sc.append(sc[-1] + torch.log(m))
    endp = torch.einsum('ps,ps->p', al[-1], chi[:, :, e_col])
    ll = torch.log(endp) + sc[-1]
    N = torch.zeros(P, n, n, dtype=F64, device=dev)
    cM, cI, cD = (torch.zeros(P * G * k, dtype=F64, device=dev) for k in (441, 21, 21))
    w = torch.zeros(P, n, dtype=F64, device=dev)
    ws = torch.zeros(P, dtype=F64, device=dev)
    for c in range(top, -1, -1):                     # w: e b of the column after c, or the step to End
        at_end = (c == L)[:, None]
        w = torch.where(at_end, torch.nn.functional.one_hot(torch.tensor(e_col, device=dev), n).to(F64), w)
        ws = torch.where(at_end[:, 0], torch.zeros_like(ws), ws)
        live = (c <= L).to(F64)
        g = torch.exp((sc[c] + ws - ll) * live) * live
        N += torch.einsum('ps,pk->psk', al[c], w) * g[:, None, None]
        b = torch.einsum('psk,pk->ps', chi, w)
        if c:
            ga = al[c] * b * g[:, None]
            for ty, acc, width, code in ((M, cM, 441, anc[:, c - 1] * 21 + des[:, c - 1]), (I, cI, 21, des[:, c - 1]),
                                         (D, cD, 21, anc[:, c - 1])):
                ks = (st_t == ty).nonzero()[:, 0]
                acc.index_add_(0, ((pr[:, None] * G + gr_t[ks]) * width + code[:, None]).reshape(-1), ga[:, ks].reshape(-1))
            w = b * em[c - 1]
            m = w.sum(1)
            m = torch.where(m > 0, m, torch.ones_like(m))
            w, ws = w / m[:, None], ws + torch.log(m)
    return {'log_p': ll, 'n_trans': N * chi, 'cnt_M': cM.view(P, G, 21, 21), 'cnt_I': cI.view(P, G, 21),
            'cnt_D': cD.view(P, G, 21)}


def _score_gradients(q, r):
    """Gradients of -sum log P through the model's builders: dL/dtheta = sum n dlog(theta)."""
    q = {k: v.detach().requires_grad_() for k, v in q.items()}
    tabs = _mixdom2_model(q)[:4]
    w = 0.0
    for tab, n in zip(tabs, (r['n_trans'], r['cnt_M'], r['cnt_I'], r['cnt_D'])):
        w = w + (n * torch.log(torch.where(tab > 0, tab, torch.ones_like(tab)))).sum()
    g = torch.autograd.grad(-w, [q[k] for k in _GRAD_ARGS])
    return dict(zip(_GRAD_ARGS, g))


def _bin(n):
    """The padded side of n residues: the least of 4, 4 * 1.2, ... (rounded) that holds them."""
    v = 4.0
    while round(v) < n:
        v *= 1.2
    return int(round(v))


def exact(case, seed):
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    s, kind = _inputs(case, seed), case['kind']
    p = s['p']
    if case.get('K', 0):
        q = _tensors(p, s['ts'], dev)
        *tabs, sub = _mixdom2_model(q)
    else:
        tabs = _tkf_model(p, s['ts'], dev, floor=kind != 'posteriors')
    none = {'status': None}
    if kind == 'estep':
        r = _batched(case, s, tabs, dev)
        r.update(_class_counts(q, sub, r['cnt_M'], r['cnt_I'], r['cnt_D']))
        r.update(_dwell(q, sub, q['t'], r['class_match_counts']))
        return {**r, **none}
    if kind == 'tkf92_forward':
        return _batched(case, s, tabs, dev, want='ll')['log_p']
    if kind == 'tkf92_estep':
        r = _batched(case, s, tabs, dev)
        return {'log_p': r['log_p'], 'n_chi_diag': r['n_trans'], **_birth_death(r['n_trans'], p, s['ts'], dev), **none}
    if kind == 'banded':
        st, gr = _states(case)
        r = _lattice(st, gr, tabs, s['xs'], s['ys'], dev, want='posteriors', band=(s['centers'], case['width']))
        post, w = r.pop('posteriors'), case['width']
        rows = []
        for k, (y, c) in enumerate(zip(s['ys'], s['centers'])):
            j = torch.as_tensor(c, device=dev).long()[:, None] + torch.arange(-w, w + 1, device=dev)
            on = (j >= 0) & (j <= len(y))
            i = torch.arange(len(c), device=dev)[:, None].expand_as(j)
            rows.append(post[k][i, j.clamp(0, post.shape[2] - 1)] * on[..., None])
        return {'ll': r.pop('log_p'), **r, 'post_band': torch.cat(rows), **none}
    if kind == 'aligned_estep':
        r = _along(case, s, tabs, dev)
        return {'log_p': r['log_p'], 'n_trans': r['n_trans'], **none}
    if kind in ('grad', 'aligned_grad'):
        r = _batched(case, s, tabs, dev) if kind == 'grad' else _along(case, s, tabs, dev)
        return {'log_p': r['log_p'], **_score_gradients(q, r)}
    if kind in ('viterbi', 'sample'):
        ll = _batched(case, s, tabs, dev, want='ll', viterbi=kind == 'viterbi')['log_p']
        return {'log_p': ll, 'paths': None, 'lengths': None}
    r = _batched(case, s, tabs, dev, want='posteriors')
    lx, ly = len(s['xs'][0]), len(s['ys'][0])
    post = torch.zeros(_bin(lx) + 1, _bin(ly) + 1, 5, dtype=F64, device=dev)   # the padded shape of the table
    post[:lx + 1, :ly + 1] = r['posteriors'][0]
    return {'log_p': r['log_p'][0], 'posteriors': post, 'n_trans': r['n_trans'][0]}
