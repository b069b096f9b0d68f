"""K above 32 (up to 1024): tile appends at the running bound, radix final select, overflow retry.

Bit-exact against the oracle's unbounded strict top-K (score desc, id asc,
zero-score fill by id), on queries with duplicates, out-of-vocabulary words,
empty rows and fewer than K matching documents; through the plain path, the
pruned path and a session whose small candidate buffer overflows so that the
retry pass must answer from its final bound.
"""

import numpy as np
import pytest

from helpers import assert_same_topk, mixed_queries, pack


def test_large_k_options_checked(pkg):
    """max_k above 32 needs the tile-group kernel; 1024 is the largest K (no device needed)."""
    spec = pkg.CorpusSpec(docs=4096, vocab=500, seed=3)
    index = pkg.synthetic_index(spec)
    with pytest.raises(pkg.InvalidParam):
        pkg.Bm25Session.from_lazy(index.offsets, index.docs, index.tf, index.norm, index.idf, max_k=64, kernel=0)
    with pytest.raises(pkg.InvalidParam):
        pkg.Bm25Session.from_lazy(index.offsets, index.docs, index.tf, index.norm, index.idf, max_k=1025)


@pytest.fixture(scope='module')
def corpus(pkg, oracle_mod):
    spec = pkg.CorpusSpec(docs=200_000, vocab=20_000, seed=77, k1=1.2)
    index = pkg.synthetic_index(spec)
    data = oracle_mod.contributions(index, spec.k1)
    return index, data


def _queries(index, seed, count):
    rng = np.random.default_rng(seed)
    rows = mixed_queries(index.vocab, rng, count, 1, 12, oov=True)
    rows += [[], [index.vocab - 1], [0, 0, 0]]  # empty, a rare word (fewer than K matches), duplicates
    return pack(rows)


@pytest.mark.gpu
@pytest.mark.parametrize('kernel,tile_docs', [(5, 1024), (4, 1024), (4, 2048)])
def test_large_k_plain_matches_oracle(pkg, oracle_mod, corpus, cuda_ok, kernel, tile_docs):
    index, data = corpus
    offsets, words = _queries(index, tile_docs, 29)
    with pkg.Bm25Session.from_csc(index.offsets, index.docs, data, index.num_docs, query_capacity=64,
                                  word_capacity=1024, max_k=1024, tile_docs=tile_docs, kernel=kernel) as s:
        for k in (33, 100, 1000, 1024, 10):
            want = oracle_mod.search(index.offsets, index.docs, data, index.num_docs, offsets, words, k)
            assert_same_topk(*s.search((offsets, words), k), *want, f'k={k}')
            assert s.device_status() == 0


@pytest.mark.gpu
def test_large_k_overflow_is_retried(pkg, oracle_mod, corpus, cuda_ok):
    """A candidate buffer of 2048 per query overflows on the first pass for common words; the
    retry pass searches those queries again from their final bound and still answers exactly."""
    index, data = corpus
    df = np.diff(index.offsets)
    common = [int(x) for x in np.argsort(-df)[:6]]
    rows = [common[:2], common[2:5], [common[0]], common[1:6]]
    offsets, words = pack(rows)
    with pkg.Bm25Session.from_csc(index.offsets, index.docs, data, index.num_docs, query_capacity=8,
                                  word_capacity=64, max_k=256, candidate_capacity=2048) as s:
        for k in (100, 256):
            want = oracle_mod.search(index.offsets, index.docs, data, index.num_docs, offsets, words, k)
            assert_same_topk(*s.search((offsets, words), k), *want, f'k={k}')
            s.search_stats(reset=True)


@pytest.mark.gpu
def test_large_k_pruned_matches_oracle(pkg, oracle_mod, corpus, cuda_ok):
    index, data = corpus
    offsets, words = _queries(index, 5, 29)
    q = offsets.size - 1
    # a buffer that holds every document: no query overflows, so the flags follow tau alone
    with pkg.Bm25Session.from_csc(index.offsets, index.docs, data, index.num_docs, query_capacity=64,
                                  word_capacity=1024, max_k=1000, prune=True,
                                  candidate_capacity=index.num_docs + 2048) as s:
        for k in (100, 1000):
            want_s, want_i, full = oracle_mod.search(index.offsets, index.docs, data, index.num_docs, offsets,
                                                     words, k, full=True)
            kth = want_s[:, -1]
            for label, tau in (('kth', kth), ('0.8 kth', kth * np.float32(0.8)), ('2 kth', kth * np.float32(2)),
                               ('zero', np.zeros(q, np.float32))):
                got_s, got_i, exact = s.search_pruned((offsets, words), k, tau.astype(np.float32))
                assert_same_topk(got_s, got_i, want_s, want_i, f'k={k} {label}')
                reach = ((full >= tau[:, None]) & (full > 0)).sum(axis=1)
                assert np.array_equal(exact, np.where(~(tau > 0) | (reach >= k), 1, 0)), label
            s.set_threshold_model(None)  # safe bounds alone (term ranks 64..1024): proven, so nothing fails
            got_s, got_i, exact = s.search_learned((offsets, words), k)
            assert_same_topk(got_s, got_i, want_s, want_i, f'k={k} learned (no model)')
            assert exact.all()


def _by_k(oracle_mod, index, data, offsets, words, ks):
    """Oracle rows for a batch with a K per query, packed like bm25_search_batch."""
    out_s, out_i = [], []
    for i, k in enumerate(ks):
        o = np.array([0, offsets[i + 1] - offsets[i]], dtype=np.int64)
        w = words[offsets[i]:offsets[i + 1]]
        s, d = oracle_mod.search(index.offsets, index.docs, data, index.num_docs, o, w, int(k))
        out_s.append(s[0])
        out_i.append(d[0])
    return np.concatenate(out_s), np.concatenate(out_i)


@pytest.mark.gpu
def test_batch_with_k_per_query(pkg, oracle_mod, corpus, cuda_ok):
    """One Search of 40 queries with K drawn from {1, 10, 32, 33, 100, 1000}: packed rows equal the
    oracle's per-query top-K, through the plain path, the learned path (safe bounds and a model of
    random weights whose bounds fall back often) and the device entry point."""
    import torch
    index, data = corpus
    offsets, words = _queries(index, 11, 37)
    q = offsets.size - 1
    rng = np.random.default_rng(4)
    ks = rng.choice([1, 10, 32, 33, 100, 1000], q).astype(np.int32)
    want_s, want_i = _by_k(oracle_mod, index, data, offsets, words, ks)
    with pkg.Bm25Session.from_csc(index.offsets, index.docs, data, index.num_docs, query_capacity=64,
                                  word_capacity=1024, max_k=1000, prune=True) as s:
        got_s, got_i, koff = s.search_batch((offsets, words), ks)
        assert koff[-1] == ks.sum()
        assert_same_topk(got_s[None], got_i[None], want_s[None], want_i[None], 'batch plain')
        for model in (None, pkg.learned.ThresholdModel(pkg.learned.init_params(1, 3.0), -1.0)):
            s.set_threshold_model(model)
            got_s, got_i, koff, exact = s.search_batch((offsets, words), ks, learned=True)
            assert_same_topk(got_s[None], got_i[None], want_s[None], want_i[None], f'batch learned {model is None}')
        dev = torch.device('cuda:0')
        d = {name: torch.from_numpy(x).to(dev) for name, x in
             (('o', offsets), ('w', words), ('k', ks), ('ko', koff[:-1].copy()))}
        d_s = torch.empty(int(koff[-1]), dtype=torch.float32, device=dev)
        d_i = torch.empty(int(koff[-1]), dtype=torch.int32, device=dev)
        d_x = torch.empty(q, dtype=torch.int32, device=dev)
        for learned in (False, True):
            s.search_batch_device(d['o'].data_ptr(), d['w'].data_ptr(), d['k'].data_ptr(), d['ko'].data_ptr(), q,
                                  int(ks.max()), d_s.data_ptr(), d_i.data_ptr(), d_x.data_ptr(), learned,
                                  torch.cuda.current_stream(dev).cuda_stream)
            torch.cuda.synchronize()
            assert s.device_status() == 0
            assert_same_topk(d_s.cpu().numpy()[None], d_i.cpu().numpy()[None], want_s[None], want_i[None],
                             f'batch device learned={learned}')


@pytest.mark.gpu
def test_tune_batch_with_k_per_query_learned(pkg, oracle_mod, corpus, cuda_ok):
    """The live-session tuner on a learned batch with a K per query (as the benchmark tunes the routing
    cut): every cut answers the same bits, the fastest is kept, and the session still answers the
    oracle's rows afterwards."""
    index, data = corpus
    offsets, words = _queries(index, 11, 41)
    q = offsets.size - 1
    ks = np.random.default_rng(9).choice([10, 100, 1000], q).astype(np.int32)
    want_s, want_i = _by_k(oracle_mod, index, data, offsets, words, ks)
    with pkg.Bm25Session.from_csc(index.offsets, index.docs, data, index.num_docs, query_capacity=64,
                                  word_capacity=1024, max_k=1000, prune=True) as s:
        s.set_threshold_model(pkg.learned.ThresholdModel(pkg.learned.init_params(1, 3.0), -1.0))
        best, table = pkg.autotune.tune(s, (offsets, words), int(ks.max()), space={'prune_route': (0.2, 1.0)},
                                        learned=True, ks=ks, reps=2)
        assert len(table) == 2 and best['prune_route'] in (0.2, 1.0) and s.tuning()['prune_route'] == best['prune_route']
        got_s, got_i, _, _ = s.search_batch((offsets, words), ks, learned=True)
        assert_same_topk(got_s[None], got_i[None], want_s[None], want_i[None], 'tuned learned batch')


@pytest.mark.gpu
@pytest.mark.parametrize('k', [33, 64, 65, 1000, 1024])
def test_large_k_from_seeds_with_ties(pkg, oracle_mod, cuda_ok, k):
    """Words whose seed (the score at a stored rank) equals the K-th score, with ties past it, lists of
    exactly K and K - 1 postings, and scores over many octaves; one K and a K per query."""
    rng = np.random.default_rng(k)
    docs = 50_001
    lists = [(docs // 2, 1.0), (k, 2.0), (k - 1, 3.0), (2048, None), (1, 4.0)]
    ids = [np.sort(rng.choice(docs, size=n, replace=False)).astype(np.int32) for n, _ in lists]
    data = [np.full(n, v, np.float32) if v else np.exp2(rng.uniform(-20, 20, n)).astype(np.float32) for n, v in lists]
    indptr = np.concatenate([[0], np.cumsum([n for n, _ in lists])]).astype(np.int64)
    ids, data = np.concatenate(ids), np.concatenate(data)
    offsets, words = pack([[0], [1], [2], [3], [0, 1], [2, 3, 0], [], [4, 1], [3, 3], [4]])
    want = oracle_mod.search(indptr, ids, data, docs, offsets, words, k)
    with pkg.Bm25Session.from_csc(indptr, ids, data, docs, query_capacity=16, word_capacity=64, max_k=1024) as s:
        for _ in range(2):
            assert_same_topk(*s.search((offsets, words), k), *want, f'k={k}')
        ks = np.resize(np.array([k, 10, 32], np.int32), offsets.size - 1)
        scores, got, _ = s.search_batch((offsets, words), ks)
        start = 0
        for q, kq in enumerate(ks):
            ref = oracle_mod.search(indptr, ids, data, docs, *pack([words[offsets[q]:offsets[q + 1]].tolist()]), int(kq))
            assert_same_topk(scores[start:start + kq], got[start:start + kq], ref[0].ravel(), ref[1].ravel(), f'q={q}')
            start += kq
        assert s.device_status() == 0


@pytest.mark.gpu
def test_large_k_with_few_candidates(pkg, oracle_mod, cuda_ok):
    """Candidate counts at the edges of the whole sort (K, 256) and of the sorted list (1024), with ties
    across the K-th score, through the plain path and the safe bounds."""
    rng = np.random.default_rng(6)
    docs = 20_000
    counts = [1, 33, 34, 99, 100, 101, 255, 256, 257, 258, 1023, 1024, 1025, 3000]
    ids = [np.sort(rng.choice(docs, size=n, replace=False)).astype(np.int32) for n in counts]
    data = [rng.choice([0.5, 0.75, 3.0], n).astype(np.float32) for n in counts]
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ids, data = np.concatenate(ids), np.concatenate(data)
    rows = [[t] for t in range(len(counts))] + [[0, 6], [4, 5], [7, 7], [1, 8, 2], []]
    offsets, words = pack(rows)
    with pkg.Bm25Session.from_csc(indptr, ids, data, docs, query_capacity=32, word_capacity=64, max_k=1024,
                                  prune=True) as s:
        for k in (33, 64, 100, 255, 256, 257, 1023, 1024):
            want = oracle_mod.search(indptr, ids, data, docs, offsets, words, k)
            assert_same_topk(*s.search((offsets, words), k), *want, f'k={k}')
            assert_same_topk(*s.search_learned((offsets, words), k)[:2], *want, f'k={k} learned')
        assert s.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize('max_k', [32, 1000])
def test_batch_of_small_k_per_query(pkg, oracle_mod, corpus, cuda_ok, max_k):
    """Batches whose K are all at most 32, on the default kernel: empty queries first, in the middle and
    last, unknown words, 33 to 64 words, batches below their bucket and below the capacity, every claim
    size, through host and device buffers."""
    import torch
    index, data = corpus
    rng = np.random.default_rng(max_k)
    df = np.diff(index.offsets)
    common = [int(x) for x in np.argsort(-df)[:40]]
    rows = mixed_queries(index.vocab, rng, 48, 0, 10, oov=True)
    rows += [list(rng.integers(0, index.vocab, n)) for n in (32, 33, 63, 64)] + [common[:33], common[:1], common[:4]]
    rows = [[]] + rows[:30] + [[], [index.vocab + 7], []] + rows[30:] + [[]]  # 60 queries: a bucket of 64, a capacity of 96
    dev = torch.device('cuda:0')
    with pkg.Bm25Session.from_csc(index.offsets, index.docs, data, index.num_docs, query_capacity=96,
                                  word_capacity=2048, max_k=max_k) as s:
        for count, tuning in ((60, {}), (60, {'claim_tiles': 2, 'tail_claims': 0}), (60, {'claim_tiles': 8}),
                              (60, {'claim_tiles': 4, 'tail_claims': 0}), (3, {}), (1, {})):
            s.set_tuning(**tuning)
            part = rows[:count] if count > 3 else rows[-3:-3 + count or None]
            offsets, words = pack([[int(x) for x in r] for r in part])
            ks = rng.choice([1, 7, 10, 31, 32], count).astype(np.int32)
            want_s, want_i = _by_k(oracle_mod, index, data, offsets, words, ks)
            for _ in range(2):  # the second finds the state that the first left
                got_s, got_i, koff = s.search_batch((offsets, words), ks)
                assert_same_topk(got_s[None], got_i[None], want_s[None], want_i[None], f'{count} {tuning}')
            d = [torch.from_numpy(x).to(dev) for x in (offsets, words, ks, koff[:-1].copy())]
            d_s = torch.empty(int(koff[-1]), dtype=torch.float32, device=dev)
            d_i = torch.empty(int(koff[-1]), dtype=torch.int32, device=dev)
            s.search_batch_device(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(), count,
                                  int(ks.max()), d_s.data_ptr(), d_i.data_ptr(), None, False,
                                  torch.cuda.current_stream(dev).cuda_stream)
            torch.cuda.synchronize()
            assert s.device_status() == 0
            assert_same_topk(d_s.cpu().numpy()[None], d_i.cpu().numpy()[None], want_s[None], want_i[None],
                             f'device {count} {tuning}')


@pytest.mark.gpu
def test_batch_of_small_k_with_ties_at_the_seed(pkg, oracle_mod, cuda_ok):
    """A K per query up to 32 where the word's K-th posting score, the bound that its query starts from,
    is tied past rank K, and where a list holds exactly K, K - 1 and one posting."""
    rng = np.random.default_rng(12)
    docs = 150_001
    counts = [docs // 3, 32, 31, 10, 9, 1, 5000]
    ids = [np.sort(rng.choice(docs, size=n, replace=False)).astype(np.int32) for n in counts]
    data = [np.full(n, 1.0 + i, np.float32) for i, n in enumerate(counts)]
    data[-1] = np.exp2(rng.uniform(-20, 20, counts[-1])).astype(np.float32)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ids, data = np.concatenate(ids), np.concatenate(data)
    rows = [[0], [1], [2], [3], [4], [5], [6], [0, 1], [0, 0], [6, 0], [4, 3, 2, 1], []]
    offsets, words = pack(rows)
    with pkg.Bm25Session.from_csc(indptr, ids, data, docs, query_capacity=32, word_capacity=64, max_k=32) as s:
        for first in range(3):
            ks = np.resize(np.array([32, 10, 1][first:] + [31, 9], np.int32), len(rows))
            got_s, got_i, koff = s.search_batch((offsets, words), ks)
            for q, k in enumerate(ks):
                ref = oracle_mod.search(indptr, ids, data, docs, *pack([rows[q]]), int(k))
                assert_same_topk(got_s[koff[q]:koff[q] + k], got_i[koff[q]:koff[q] + k], ref[0].ravel(),
                                 ref[1].ravel(), f'q={q} k={k}')
