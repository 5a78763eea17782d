"""Fold-in with either walk against the CPU oracle, bit for bit: a model whose
words have short lists of topics (the walk over the words' lists), one whose
words have long ones (documents' topics or words' lists), and one with a few
long lists among short ones; requests around a chunk's length."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g
from gpupolyaurnlda_b200.serve import Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["launch", "persistent"])
@pytest.mark.parametrize("K,lists", [(50, (1, 50)), (700, (1, 160)), (700, (161, 700)), (700, (1, 170)), (2048, (700, 2048))])
def test_fold_in_walks_match_oracle(gpu_lib, oracle_lib, K, lists, mode):
    rng = np.random.default_rng(K + lists[0])
    V, n_iter = 60, 3
    n0 = np.zeros((V, K), np.uint32)
    for w in range(V):
        n = int(rng.integers(lists[0], lists[1] + 1)) if w else lists[1]
        n0[w, rng.permutation(K)[:n]] = rng.integers(1, 200, n)
    if lists == (1, 170):
        n0[V - 1, :10] = 1000000  # most of the mass in a short list
    with g.Sampler(0.1, 0.0, K, np.full(V, 5, np.uint32), buffer_size=16, max_D=4, seed=2) as s:
        s.write_counts(n0.reshape(-1))
        s.sample_phi()
        st = s.read_state(n=False, S=False)
        srv = Server(n_iter, mode=mode, slots=2, seed=9, chain=3, pool_bytes=1 << 24)
    lengths = np.array([0, 1, 2, 31, 32, 33, 63, 64, 65, 200, 1500], np.uint32)
    words = rng.integers(0, V, int(lengths.sum())).astype(np.uint32)
    ids = np.arange(len(lengths), dtype=np.uint64) + 77
    srv.submit(ids, lengths, words)
    srv.drain()
    out = srv.poll(len(ids))
    srv.close()
    order = np.argsort(out["ids"])
    ref = oracle_lib.fold_in(K, V, 0.1, st, words, lengths, ids, n_iter, seed=9, chain=3)
    assert (out["theta"][order].view(np.uint32) == ref["theta"].view(np.uint32)).all()
    assert (out["skipped"][order] == ref["skipped"]).all()
    np.testing.assert_allclose(out["ll"][order], ref["ll"], rtol=1e-9, atol=1e-9)
