"""What a user of this engine has it do, as cases that can be timed and compared.

A user's program holds one resident index per corpus (a session) and sends it query batches: a
few queries at a time through host buffers, a serving loop's uneven batches, large evaluation
batches, plain or with learned starting bounds, K from 10 to 1000.  Beside that it builds indexes
from token ids and trains the threshold model.  The corpora here are the shapes of
CONFIG_SHAPES and of the tests (Zipf tokens and lognormal lengths, or the reference's uniform
1024-term corpus), generated on the GPU by a seeded generator of this file; a corpus depends on
its shape alone, so that every state of a case uses one resident session as a program does, and
the queries (terms drawn by document frequency), their K and the training data come from the seed.
"""

import collections
import importlib
import math

import numpy as np
import torch

B200 = importlib.import_module('bm25-npu_b200')
DEV = 'cuda:0'
_stream = []  # the program's own stream for device-resident calls


def _own_stream():
    if not _stream:
        _stream.append(torch.cuda.Stream(DEV))
    return _stream[0].cuda_stream


def _corpus_fields(docs, vocab, zipf=1.1, mean=60.0, sigma=0.5, k1=1.5):
    return {'docs': docs, 'vocab': vocab, 'zipf': zipf, 'mean': mean, 'sigma': sigma, 'k1': k1}


SYNTHETIC_10M = _corpus_fields(10_000_000, 1_000_000)
REFERENCE_10M = _corpus_fields(10_000_000, 1024, zipf=0.0, mean=32.0, sigma=-16.0, k1=1.2)
PASSAGES_8P8M = _corpus_fields(8_800_000, 2_500_000, zipf=1.05, mean=56.0)
BLOCKMAX_4P2M = _corpus_fields(4_200_000, 1_000_000, mean=80.0)


def listed():
    return [
        # an interactive lookup in a small collection: one query through host buffers, all latency
        dict(name='small_one_query', kind='search', **_corpus_fields(8192, 30_000), queries=1, lo=3, hi=3, ks='10'),
        # a mid-sized collection with odd sizes: an evaluation batch with deep results (K 1000)
        dict(name='deep_results_1m', kind='search', **_corpus_fields(1_000_003, 300_000), queries=37, lo=1, hi=12,
             ks='1000'),
        # the engine's headline call: 8 queries of 3 terms on 10M documents through host buffers
        dict(name='plain_10m', kind='search', **SYNTHETIC_10M, queries=8, lo=3, hi=3, ks='10'),
        # the same call with a trained threshold model
        dict(name='learned_10m', kind='learned', **SYNTHETIC_10M, queries=8, lo=3, hi=3, ks='10'),
        # one round of a serving loop: the queries that arrived meanwhile, 1-16 terms, mixed K
        dict(name='serve_round_10m', kind='batch_learned', **SYNTHETIC_10M, queries=23, lo=1, hi=16, ks='10,100,1000'),
        # queries and results kept in HBM, on the reference's own corpus shape (uniform terms)
        dict(name='device_reference_10m', kind='device', **REFERENCE_10M, queries=8, lo=3, hi=3, ks='10'),
        # the batched mix: 256 uneven queries in one call, plain and learned
        dict(name='mix_plain_8p8m', kind='batch', **PASSAGES_8P8M, queries=256, lo=2, hi=12, ks='10,100,1000'),
        dict(name='mix_learned_8p8m', kind='batch_learned', **PASSAGES_8P8M, queries=256, lo=2, hi=12,
             ks='10,100,1000'),
        # an offline evaluation in device-resident batches with a trained model
        dict(name='blockmax_4p2m', kind='device_learned', **BLOCKMAX_4P2M, queries=250, lo=2, hi=10, ks='10,100'),
        # a shard or a tenant of a larger service: medium batch, plain, odd sizes
        dict(name='tenant_262k', kind='batch', **_corpus_fields(262_147, 100_000), queries=50, lo=1, hi=8, ks='10,32'),
        # a new index from token ids (host arrays in and out)
        dict(name='build_index_200k', kind='build', **_corpus_fields(200_003, 200_000)),
        # the threshold model's training loop
        dict(name='train_model', kind='train', samples=20_000, steps=60, batch=4096),
    ]


def draw(rng):
    kind = rng.choice(['search', 'search', 'learned', 'device', 'batch', 'batch_learned', 'device_learned', 'build',
                       'train'])
    if kind == 'train':
        return {'kind': kind, 'samples': rng.randint(5_000, 20_000), 'steps': rng.randint(20, 60),
                'batch': int(math.exp(rng.uniform(math.log(256), math.log(4097))))}
    top = 200_000 if kind == 'build' else 9_999_999
    docs = int(math.exp(rng.uniform(math.log(8192), math.log(top))))
    if rng.random() < 0.15:
        shape = _corpus_fields(docs, 1024, zipf=0.0, mean=32.0, sigma=-16.0, k1=1.2)
    else:
        vocab = int(math.exp(rng.uniform(math.log(30_000), math.log(1_000_000))))
        shape = _corpus_fields(docs, vocab, zipf=rng.choice([1.05, 1.1]), mean=rng.choice([56.0, 60.0, 80.0]))
    if kind == 'build':
        return dict(kind=kind, **shape)
    queries = int(math.exp(rng.uniform(0.0, math.log(257)))) if docs < 8_000_000 else rng.randint(1, 32)
    lo = rng.randint(1, 3)
    hi = rng.randint(lo, 12)
    if kind.endswith('_learned') or kind == 'batch':
        ks = rng.choice(['10,100', '10,100,1000', '10,32', '10'])
    else:
        ks = rng.choice(['10', '10', '32', '1', '100', '1000'])
    return dict(kind=kind, **shape, queries=queries, lo=lo, hi=hi, ks=ks)


# ---- corpora -------------------------------------------------------------------------------------

def _zipf(case):
    p = np.arange(1, case['vocab'] + 1, dtype=np.float64) ** -case['zipf']
    return p / p.sum()


def _tokens(case, seed):
    """Document lengths int64 [docs] and the tokens' document and term ids (GPU, seeded)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n, mean, sigma = case['docs'], case['mean'], case['sigma']
    if sigma < 0:
        w = int(round(-sigma))
        length = torch.randint(int(mean) - w, int(mean) + w + 1, (n,), generator=g, device=DEV)
    else:
        z = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
        length = torch.exp(z * sigma + (math.log(mean) - sigma * sigma / 2)).round().clamp(1, 4096).long()
    cdf = torch.from_numpy(np.cumsum(_zipf(case))).to(DEV)
    total = int(length.sum())
    u = torch.rand(total, generator=g, device=DEV, dtype=torch.float64)
    term = torch.searchsorted(cdf, u, right=True).clamp_(max=case['vocab'] - 1)
    del u
    return length, torch.repeat_interleave(torch.arange(n, device=DEV), length), term


def _documents(case, seed):
    """The corpus's documents in an order of the seed, with term ids in an order of the seed."""
    length, doc, term = _tokens(case, 20261203)
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    place = torch.randperm(case['docs'], generator=g, device=DEV)
    moved = torch.empty_like(length)
    moved[place] = length
    doc, at = torch.sort(place[doc], stable=True)
    return moved, doc, torch.randperm(case['vocab'], generator=g, device=DEV)[term[at]]


_corpora = collections.OrderedDict()  # the latest corpora: CSC on the host
_sessions = collections.OrderedDict()  # resident sessions (and their models), the latest ones
_SHAPE = ('docs', 'vocab', 'zipf', 'mean', 'sigma', 'k1')


def _latest(cache, key, make, most):
    if key in cache:
        cache.move_to_end(key)
        return cache[key]
    while len(cache) >= most:
        cache.popitem(last=False)
    cache[key] = make()
    return cache[key]


def _make_corpus(case):
    length, doc, term = _tokens(case, 20261203)
    key = term.bitwise_left_shift_(32).bitwise_or_(doc)
    del doc, term
    key = torch.sort(key).values
    first = torch.ones(key.numel(), dtype=torch.bool, device=DEV)
    torch.ne(key[1:], key[:-1], out=first[1:])
    start = first.nonzero().flatten()
    del first
    tf = torch.diff(start, append=torch.tensor([key.numel()], device=DEV)).float()
    key = key[start]
    del start
    doc, term = key.bitwise_and(0xffffffff), key.bitwise_right_shift(32)
    del key
    n, k1, b = case['docs'], case['k1'], 0.75
    df = torch.bincount(term, minlength=case['vocab'])
    idf = torch.log1p((n - df.double() + 0.5) / (df.double() + 0.5)).float()
    ln = length.double()
    norm = (k1 * (1 - b + b * ln / ln.mean())).float()
    data = idf[term] * (tf * np.float32(k1 + 1.0)) / (tf + norm[doc])
    indptr = torch.zeros(case['vocab'] + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = df.cumsum(0)
    out = indptr.cpu().numpy(), doc.int().cpu().numpy(), data.cpu().numpy()
    del doc, term, tf, data, df
    torch.cuda.empty_cache()
    return out


def _corpus(case):
    """Eager CSC of the case's corpus (host): indptr int64, doc ids int32, scores float32."""
    return _latest(_corpora, tuple(case[f] for f in _SHAPE), lambda: _make_corpus(case), 2)


def _queries(indptr, count, lo, hi, rng):
    """Packed queries of lo..hi distinct terms drawn by document frequency."""
    present = int((np.diff(indptr) > 0).sum())
    rows = []
    for _ in range(count):
        n = min(int(rng.integers(lo, hi + 1)), present)
        row = []
        while len(row) < n:
            for t in np.searchsorted(indptr, rng.integers(0, indptr[-1], 4 * n), side='right') - 1:
                if int(t) not in row and len(row) < n:
                    row.append(int(t))
        rows.append(row)
    offsets = np.zeros(count + 1, dtype=np.int64)
    np.cumsum([len(r) for r in rows], out=offsets[1:])
    return offsets, np.array([t for r in rows for t in r], dtype=np.int32)


# ---- sessions and threshold models ---------------------------------------------------------------

def _ks(case):
    return [int(k) for k in case['ks'].split(',')]


def _fit_model(session, indptr, case):
    """A threshold model for the session, trained in 64 bits on queries of the case's shape: the
    weights that a program with learned bounds loads."""
    rng = np.random.default_rng(77)
    cap, rounds = case['queries'], max(2, min(256, 2048 // case['queries']))
    feats, logk = [], []
    for _ in range(rounds):
        for k in _ks(case):
            offsets, words = (torch.from_numpy(x).to(DEV) for x in _queries(indptr, cap, case['lo'], case['hi'], rng))
            scores = torch.empty((cap, k), dtype=torch.float32, device=DEV)
            ids = torch.empty((cap, k), dtype=torch.int32, device=DEV)
            f = torch.empty((cap, 32), dtype=torch.float32, device=DEV)
            torch.cuda.synchronize()
            stream = _own_stream()
            session.search_device(offsets.data_ptr(), words.data_ptr(), cap, k, scores.data_ptr(), ids.data_ptr(),
                                  stream)
            session.query_features_device(offsets.data_ptr(), words.data_ptr(), cap, k, f.data_ptr(), None, stream)
            torch.cuda.synchronize()
            kth = scores[:, k - 1].double()
            feats.append(f[kth > 0].double())
            logk.append(kth[kth > 0].log())
    x, y = torch.cat(feats), torch.cat(logk)
    if y.numel() < 8:
        return None  # hardly any query reaches K matches: the safe bounds alone
    w = [torch.from_numpy(a).to(DEV).requires_grad_() for a in (
        rng.normal(0, math.sqrt(2 / 32), (64, 32)), np.zeros(64), rng.normal(0, math.sqrt(2 / 64), (64, 64)),
        np.zeros(64), rng.normal(0, 0.125, 64), np.full(1, float(y.mean())))]

    def predict(v):
        h = torch.relu(torch.relu(v @ w[0].T + w[1]) @ w[2].T + w[3])
        return h @ w[4] + w[5]

    held = torch.arange(y.numel(), device=DEV) % 5 == 0
    opt = torch.optim.Adam(w, lr=3e-3)
    for _ in range(300):
        opt.zero_grad()
        e = predict(x[~held]) - y[~held]
        (torch.where(e > 0, 4.0, 1.0) * e * e).mean().backward()
        opt.step()
    with torch.no_grad():
        margin = float(torch.quantile(predict(x[held]) - y[held], 0.98))
    params = torch.cat([a.detach().reshape(-1) for a in w]).float().cpu().numpy()
    return B200.learned.ThresholdModel(params, margin)


def _make_session(case):
    indptr, docs, data = _corpus(case)
    learned = case['kind'].endswith('learned')
    both = learned or case['kind'] == 'batch'  # a service that offers both keeps one session
    session = B200.Bm25Session.from_csc(
        indptr, docs, data, case['docs'], query_capacity=case['queries'],
        word_capacity=case['queries'] * case['hi'], max_k=min(max(_ks(case)), case['docs']), prune=both)
    if both:
        session.set_threshold_model(_fit_model(session, indptr, case))
    return session, indptr


def _session(case):
    both = case['kind'].endswith('learned') or case['kind'] == 'batch'
    key = tuple(case[f] for f in _SHAPE + ('queries', 'lo', 'hi', 'ks')) + (both,)
    return _latest(_sessions, key, lambda: _make_session(case), 10)


# ---- the cases -----------------------------------------------------------------------------------

def _query_inputs(case, indptr, seed):
    rng = np.random.default_rng(seed)
    offsets, words = _queries(indptr, case['queries'], case['lo'], case['hi'], rng)
    ks = np.resize([min(k, case['docs']) for k in _ks(case)], case['queries']).astype(np.int32)
    rng.shuffle(ks)
    return offsets, words, ks


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.lognormal(-0.3, 0.4, (case['samples'], 32)).astype(np.float32)
    x[:, 27] = 1.0
    x[:, 28:] = 0.0
    y = 0.9 * x[:, 0] + 0.5 * x[:, 17] + 0.2 * np.sqrt(x[:, 4]) + 0.1 * rng.standard_normal(case['samples'])
    return x, y.astype(np.float32)


def prepare(case, seed):
    kind = case['kind']
    if kind == 'train':
        x, y = _train_inputs(case, seed)
        return {'kind': kind, 'x': x, 'y': y, 'steps': case['steps'], 'batch': case['batch'], 'seed': seed % 1000}
    if kind == 'build':
        length, _, term = _documents(case, seed)
        offsets = np.zeros(case['docs'] + 1, dtype=np.int64)
        offsets[1:] = length.cumsum(0).cpu().numpy()
        return {'kind': kind, 'offsets': offsets, 'tokens': term.int().cpu().numpy(), 'vocab': case['vocab'],
                'k1': case['k1']}
    session, indptr = _session(case)
    offsets, words, ks = _query_inputs(case, indptr, seed)
    state = {'kind': kind, 'session': session, 'queries': (offsets, words), 'ks': ks, 'k': int(ks[0])}
    if kind.startswith('device'):
        q = case['queries']
        total = int(ks.sum()) if kind == 'device_learned' else q * int(ks[0])
        kout = np.cumsum(ks, dtype=np.int64) - ks
        state['in'] = [torch.from_numpy(a).to(DEV) for a in (offsets, words, ks, kout)]
        state['kmax'] = int(ks.max())
        state['scores'] = torch.empty(total, dtype=torch.float32, device=DEV)
        state['ids'] = torch.empty(total, dtype=torch.int32, device=DEV)
        state['exact'] = torch.empty(q, dtype=torch.int32, device=DEV)
        torch.cuda.synchronize()
    return state


def run(state):
    kind = state['kind']
    if kind == 'search':
        return state['session'].search(state['queries'], state['k'])
    if kind == 'learned':
        return state['session'].search_learned(state['queries'], state['k'])
    if kind in ('batch', 'batch_learned'):
        return state['session'].search_batch(state['queries'], state['ks'], learned=kind == 'batch_learned')
    if kind == 'train':
        return B200.learned.train(state['x'], state['y'], steps=state['steps'], batch=state['batch'],
                                  seed=state['seed'])
    if kind == 'build':
        index = B200.build_index(state['offsets'], state['tokens'], state['vocab'], k1=state['k1'])
        return {'offsets': index.offsets, 'docs': index.docs, 'tf': index.tf, 'norm': index.norm, 'idf': index.idf}
    offsets, words, ks, kout = state['in']
    stream = _own_stream()
    if kind == 'device':
        state['session'].search_device(offsets.data_ptr(), words.data_ptr(), offsets.numel() - 1, state['k'],
                                       state['scores'].data_ptr(), state['ids'].data_ptr(), stream)
        return state['scores'], state['ids']
    state['session'].search_batch_device(offsets.data_ptr(), words.data_ptr(), ks.data_ptr(), kout.data_ptr(),
                                         offsets.numel() - 1, state['kmax'], state['scores'].data_ptr(),
                                         state['ids'].data_ptr(), state['exact'].data_ptr(), True, stream)
    return state['scores'], state['ids'], state['exact']


def work(case):
    """Bytes: the distinct posting lists that the queries name (8 bytes a posting, in expectation:
    terms drawn by document frequency), once each, and the results; operations: one addition a
    posting and query, or the network's multiply-adds."""
    kind = case['kind']
    if kind == 'train':
        macs = 32 * 64 + 64 * 64 + 64
        rows = float(case['steps']) * min(case['batch'], case['samples'])
        return {'bytes': case['samples'] * 33 * 4 + rows * 33 * 4, 'flops': rows * macs * 2 * 3}
    if case['sigma'] < 0:
        length = case['mean'] + np.linspace(case['sigma'], -case['sigma'], 33)
    else:
        z = np.array([math.sqrt(2) * x for x in np.polynomial.hermite.hermgauss(9)[0]])
        z_w = np.polynomial.hermite.hermgauss(9)[1] / math.sqrt(math.pi)
        length = case['mean'] * np.exp(z * case['sigma'] - case['sigma'] ** 2 / 2)
    weight = np.full(length.size, 1 / length.size) if case['sigma'] < 0 else z_w
    p = _zipf(case)
    df = np.zeros_like(p)
    for x, w in zip(length, weight):
        df += w * -np.expm1(x * np.log1p(-p))
    df *= case['docs']
    if kind == 'build':
        tokens = case['docs'] * case['mean']
        return {'bytes': tokens * 4 + case['docs'] * 12 + df.sum() * 8 + case['vocab'] * 12, 'flops': 0}
    words = case['queries'] * (case['lo'] + case['hi']) / 2
    share = df / df.sum()
    once = float((df * -np.expm1(words * np.log1p(-share))).sum())
    results = case['queries'] * sum(_ks(case)) / len(_ks(case))
    return {'bytes': once * 8 + results * 8, 'flops': float((df * share).sum()) * words}


# ---- the same outputs in 64 bits ------------------------------------------------------------------

def _exact_search(case, seed):
    indptr, docs, data = _corpus(case)
    offsets, words, ks = _query_inputs(case, indptr, seed)
    mixed = case['kind'] in ('batch', 'batch_learned', 'device_learned')
    top = []
    for q in range(case['queries']):
        score = torch.zeros(case['docs'], dtype=torch.float64, device=DEV)
        for t in words[offsets[q]:offsets[q + 1]]:
            a, b = int(indptr[t]), int(indptr[t + 1])
            score.index_add_(0, torch.from_numpy(docs[a:b]).to(DEV), torch.from_numpy(data[a:b]).to(DEV).double())
        top.append(torch.topk(score, int(ks[q]) if mixed else int(ks[0])).values.cpu())
    if mixed:
        scores = torch.cat(top)
        return (scores, None, None, None) if case['kind'] == 'batch_learned' else (scores, None, None)
    if case['kind'] == 'device':
        return torch.cat(top), None
    return (torch.stack(top), None, None) if case['kind'] == 'learned' else (torch.stack(top), None)


def _exact_build(case, seed):
    length, doc, term = _documents(case, seed)
    key, count = torch.unique(term.bitwise_left_shift(32).bitwise_or(doc), return_counts=True)
    df = torch.bincount(key.bitwise_right_shift(32), minlength=case['vocab']).double()
    ln, n, b = length.double(), case['docs'], 0.75
    return {'offsets': None, 'docs': None, 'tf': count.double(), 'norm': case['k1'] * (1 - b + b * ln / ln.mean()),
            'idf': torch.log1p((n - df + 0.5) / (df + 0.5))}


def _exact_train(case, seed):
    x, y = (torch.from_numpy(a).to(DEV).double() for a in _train_inputs(case, seed))
    seed = seed % 1000
    rng = np.random.default_rng(seed)
    w = [rng.normal(0.0, np.sqrt(2.0 / 32), (64, 32)), np.zeros(64), rng.normal(0.0, np.sqrt(2.0 / 64), (64, 64)),
         np.zeros(64), rng.normal(0.0, np.sqrt(1.0 / 64), 64), None]
    w[5] = np.full(1, float(y.mean()))
    w = [torch.from_numpy(a.astype(np.float32)).to(DEV).double() for a in w]
    m, v = [torch.zeros_like(a) for a in w], [torch.zeros_like(a) for a in w]
    picks = np.random.default_rng(seed + 1)
    batch, losses = min(case['batch'], case['samples']), []
    for step in range(1, case['steps'] + 1):
        at = torch.from_numpy(picks.integers(0, case['samples'], batch)).to(DEV)
        xb, yb = x[at], y[at]
        z1 = xb @ w[0].T + w[1]
        h1 = z1.relu()
        z2 = h1 @ w[2].T + w[3]
        h2 = z2.relu()
        e = h2 @ w[4] + w[5] - yb
        over = torch.where(e > 0, 4.0, 1.0).double()
        losses.append((over * e * e).mean())
        dy = 2 * over * e / batch
        d2 = dy[:, None] * w[4] * (z2 > 0)
        d1 = (d2 @ w[2]) * (z1 > 0)
        grads = [d1.T @ xb, d1.sum(0), d2.T @ h1, d2.sum(0), h2.T @ dy, dy.sum().reshape(1)]
        for a, ma, va, g in zip(w, m, v, grads):
            ma.mul_(0.9).add_(0.1 * g)
            va.mul_(0.999).add_(0.001 * g * g)
            a.sub_(2e-3 * ma / (1 - 0.9 ** step) / ((va / (1 - 0.999 ** step)).sqrt() + 1e-8))
    return torch.cat([a.reshape(-1) for a in w]), torch.stack(losses)


def exact(case, seed):
    """What run() computes, in 64 bits (None for ids, flags and offsets: whole numbers)."""
    if case['kind'] == 'train':
        return _exact_train(case, seed)
    if case['kind'] == 'build':
        return _exact_build(case, seed)
    return _exact_search(case, seed)
