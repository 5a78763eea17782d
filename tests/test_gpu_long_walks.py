"""The large-K sweep's lists in shared memory, walked from the document's side or
the word's, against the CPU oracle, bit for bit: words with lists of every
length around the steps of the walk (32 entries, 128 of which lanes read ahead),
around the documents' numbers of topics, where the walk changes sides, and of
every topic; lists with and without their q values in shared memory.  And that
short lists are walked: a document of many topics takes much longer over words
with all topics than over words with one."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu

LISTS = [0, 1, 2, 31, 32, 33, 64, 127, 128, 129, 160, 256, 400, 560, 600, 640, 700, 1000, 1500, 2000]


@pytest.mark.parametrize("K", [2049, 7000, 9000, 20000])
def test_walks_match_oracle(gpu_lib, oracle_lib, K):
    rng = np.random.default_rng(K)
    lists = [n for n in LISTS if n <= K] + [K]
    V = len(lists)
    n0 = np.zeros((V, K), np.uint32)
    for w, n in enumerate(lists):  # (a Poisson draw of 40 or more is positive but for e^-40)
        n0[w, rng.permutation(K)[:n]] = rng.integers(40, 90, n)
    d_len = np.array([600, 650, 1200, 2000, 513, 20, 700], np.uint32)
    z = np.concatenate([rng.permutation(K)[:L] for L in d_len]).astype(np.uint32)
    N = len(z)
    w = rng.integers(0, V, N).astype(np.uint32)
    alpha = 0.02
    with g.Sampler(alpha, 0.0, K, np.full(V, 10, np.uint32), buffer_size=16, max_D=4, seed=5,
                   flags=g.GPULDA_FLAG_LOGLIK) as s:
        s.write_counts(n0.reshape(-1))
        s.corpus_load(z.copy(), w, d_len)
        s.corpus_sweep(1)
        got = s.corpus_z()
        n1 = s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"]
        c = s.counters()
        ll, skipped = s.loglik()
    phi = oracle_lib.phi_step(K, V, 0.0, n0.reshape(-1).copy(), 0, 5, 0)
    assert [int(x) for x in phi["nnz"]] == lists, "the lists have other lengths than meant"
    want = z.copy()
    r = oracle_lib.z_sweep(K, V, alpha, phi, w, want, d_len, 0, key0=5, want_ll=True)
    assert (got == want).all(), f"{(got != want).sum()} topics differ"
    assert (n1 == np.bincount(w.astype(np.int64) * K + want, minlength=K * V)).all()
    assert c["sparse_work"] == int(r["stats"][2]) and c["sparse_draws"] == int(r["stats"][3])
    assert skipped == r["ll_skipped"]
    assert abs(ll - r["ll"]) <= 1e-4 * abs(r["ll"])


def _sweep_ms(K, V, topics, L):
    rng = np.random.default_rng(1)
    n0 = np.zeros((V, K), np.uint32)
    for w in range(V):
        n0[w, rng.permutation(K)[:topics]] = 50
    z, w = rng.permutation(K)[:L].astype(np.uint32), rng.integers(0, V, L).astype(np.uint32)
    best = 1e9
    with g.Sampler(0.02, 0.0, K, np.full(V, 10, np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        for _ in range(4):
            s.write_counts(n0.reshape(-1))
            s.corpus_load(z, w, np.array([L], np.uint32))
            s.corpus_sweep(1)
            best = min(best, s.kernel_times()["z_sweep"])
    return best


def test_short_word_lists_are_walked(gpu_lib):
    short, full = _sweep_ms(8192, 64, 1, 6000), _sweep_ms(8192, 64, 8192, 6000)
    assert short < 0.6 * full, f"{short:.1f} ms over words with one topic, {full:.1f} with all"
