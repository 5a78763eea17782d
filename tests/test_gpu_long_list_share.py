"""Which of the two sweeps up to K = 2048 takes a corpus depends on how long its
words' long lists are, not only on how many tokens they have: 5 % of the tokens
in lists of 2,000 entries go to the sweep over the shorter side (the other took
1.6 times as long).  And the sweep over the words' lists with long ones among
them, where nearly all tokens' words have short ones, against the CPU oracle."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


def _sweep_ms(K, share):
    """z sweep of 30,000 documents of 100 tokens; 20 words have lists of K
    entries and that share of the tokens, the others lists of 30."""
    rng = np.random.default_rng(1)
    V, D, L, long = 4000, 30000, 100, 20
    n0 = np.zeros((V, K), np.uint32)
    n0[:long] = rng.integers(20, 60, (long, K))
    each = int(n0[:long].sum() * (1 - share) / share / (V - long) / 30)
    for w in range(long, V):
        n0[w, rng.integers(0, K, 30)] = each
    N = D * L
    w = np.where(rng.random(N) < share, rng.integers(0, long, N), rng.integers(long, V, N)).astype(np.uint32)
    topics = rng.integers(0, K, (D, 3))
    z = topics[np.repeat(np.arange(D), L), rng.integers(0, 3, N)].astype(np.uint32)
    best = 1e9
    with g.Sampler(0.05, 0.0, K, np.bincount(w, minlength=V).astype(np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        for _ in range(4):
            s.write_counts(n0.reshape(-1))
            s.corpus_load(z, w, np.full(D, L, np.uint32))
            s.corpus_sweep(1)
            best = min(best, s.kernel_times()["z_sweep"])
    return best


def test_few_tokens_in_very_long_lists(gpu_lib):
    some, many = _sweep_ms(2000, 0.05), _sweep_ms(2000, 0.3)
    assert some < 1.3 * many, f"{some:.2f} ms with 5 % of the tokens in long lists, {many:.2f} with 30 %"


@pytest.mark.parametrize("docs", ["four to a warp", "one to a warp"])
@pytest.mark.parametrize("K", [333, 1000, 2048])
def test_long_lists_among_short_ones(gpu_lib, oracle_lib, K, docs):
    rng = np.random.default_rng(K)
    lists = [n for n in (160, 161, 192, 193, 320, 321, 640, 641, 1000, 2047) if n <= K] + [K]
    V = len(lists) + 1
    n0 = np.zeros((V, K), np.uint32)
    n0[V - 1, rng.permutation(K)[:5]] = 100000000  # nearly all tokens by the model
    for w, n in enumerate(lists):
        n0[w, rng.permutation(K)[:n]] = rng.integers(40, 90, n)
    d_len = np.concatenate([[0, 1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40] * 1950 + [3]] if docs[0] == "f" else
                           [[0, 1, 5, 31, 32, 33, 64, 100, 257, 1200]]).astype(np.uint32)
    N = int(d_len.sum())
    w = rng.integers(0, V, N).astype(np.uint32)
    z = rng.integers(0, K, N).astype(np.uint32)
    with g.Sampler(0.1, 0.0, K, np.full(V, 10, np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        s.write_counts(n0.reshape(-1))
        s.corpus_load(z.copy(), w, d_len)
        s.corpus_sweep(1)
        got = s.corpus_z()
        n1 = s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"]
        c = s.counters()
    phi = oracle_lib.phi_step(K, V, 0.0, n0.reshape(-1).copy(), 0, 5, 0)
    assert [int(x) for x in phi["nnz"][:len(lists)]] == lists, "the lists have other lengths than meant"
    r = oracle_lib.z_sweep(K, V, 0.1, phi, w, z, d_len, 0, key0=5)
    assert (got == z).all(), f"{(got != z).sum()} topics differ"
    assert (n1 == np.bincount(w.astype(np.int64) * K + z, minlength=K * V)).all()
    assert c["sparse_work"] == int(r["stats"][2]) and c["sparse_draws"] == int(r["stats"][3])
