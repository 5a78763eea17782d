"""The sweep over the words' lists against the CPU oracle, bit for bit: lists of
every length around the steps of their layout and walk (32, 64, 96, 128, 160
entries, and longer ones, which take the walk out of line), documents of no
and one token and around a chunk's length, four to a warp and one to a warp, a
number of documents that is no multiple of four; and the same corpus with so
many long lists that the other sweep takes it."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu

LISTS = [0, 1, 2, 3, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 159, 160, 161, 191, 192, 193, 257, 320, 321,
         640, 641, 1000, 2047, 2048]


@pytest.mark.parametrize("mostly", ["short", "long"])
@pytest.mark.parametrize("docs", ["four to a warp", "one to a warp"])
@pytest.mark.parametrize("K", [1, 20, 161, 333, 1000, 2048])
def test_word_sweep_matches_oracle(gpu_lib, oracle_lib, K, docs, mostly):
    rng = np.random.default_rng(K)
    lists = [n for n in LISTS if n <= K] + [K]
    V = len(lists) + 1
    n0 = np.zeros((V, K), np.uint32)
    # the last word has few topics and, where short lists are to prevail, most of the tokens
    n0[V - 1, rng.permutation(K)[:min(K, 5)]] = 4000000 if mostly == "short" else 50
    for w, n in enumerate(lists):
        n0[w, rng.permutation(K)[:n]] = rng.integers(40, 90, n)
    # four to a warp: a document's chain is short beside the whole sweep's time
    d_len = np.concatenate([[0, 1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40] * 1950 + [3]] if docs[0] == "f" else
                           [[0, 1, 5, 31, 32, 33, 64, 100, 257, 1200]]).astype(np.uint32)
    N = int(d_len.sum())
    w = rng.integers(0, V, N).astype(np.uint32)
    z = rng.integers(0, K, N).astype(np.uint32)
    alpha, beta = 0.1, 0.0
    counts = np.full(V, 10, np.uint32)
    with g.Sampler(alpha, beta, K, counts, buffer_size=16, max_D=4, seed=5, flags=g.GPULDA_FLAG_LOGLIK) as s:
        s.write_counts(n0.reshape(-1))
        s.corpus_load(z.copy(), w, d_len)
        s.corpus_sweep(1)
        got = s.corpus_z()
        n1 = s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"]
        c = s.counters()
        ll, skipped = s.loglik()
    phi = oracle_lib.phi_step(K, V, beta, n0.reshape(-1).copy(), 0, 5, 0)
    assert [int(x) for x in phi["nnz"][:len(lists)]] == lists, "the lists have other lengths than meant"
    want = z.copy()
    r = oracle_lib.z_sweep(K, V, alpha, phi, w, want, d_len, 0, key0=5, want_ll=True)
    assert (got == want).all(), f"{(got != want).sum()} topics differ"
    assert (n1 == np.bincount(w.astype(np.int64) * K + want, minlength=K * V)).all()
    assert c["tokens"] == N and c["docs"] == len(d_len)
    assert c["sparse_work"] == int(r["stats"][2]) and c["sparse_draws"] == int(r["stats"][3])
    assert skipped == r["ll_skipped"]
    assert abs(ll - r["ll"]) <= 1e-4 * abs(r["ll"])
