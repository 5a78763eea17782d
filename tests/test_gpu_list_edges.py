"""Edges of the large-K sweep's document lists against the CPU oracle, bit for
bit: documents around every step of the list's slots per lane (32 entries
each), around its capacity of 512 entries, and beyond it, where a document is
handed on in the middle to the lists in shared memory; the smallest and largest
K of the path; documents of no and one token."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 64, 65, 95, 97, 128, 129, 193, 257, 470, 480, 481, 511, 512, 513, 545, 640, 1500]


@pytest.mark.parametrize("K,V", [(2049, 300), (4096, 40), (32768, 40)])
def test_list_edges_match_oracle(gpu_lib, oracle_lib, K, V):
    rng = np.random.default_rng(K)
    d_len = np.array(LENGTHS * 2, np.uint32)
    half = int(sum(LENGTHS))
    # first copies: topics all distinct where K allows; second: few topics
    z = np.concatenate([rng.permutation(K)[:L] if L <= K else rng.integers(0, K, L) for L in LENGTHS] +
                       [rng.integers(0, max(1, L // 4), L) % K for L in LENGTHS]).astype(np.uint32)
    assert len(z) == 2 * half
    w = rng.integers(0, V, len(z)).astype(np.uint32)
    counts = np.sort(np.bincount(w, minlength=V).astype(np.uint32))[::-1].copy()
    ch = oracle_lib.Chain(K, 0.05, 0.01, counts, seed=11)
    z_orc = z.copy()
    with g.Sampler(0.05, 0.01, K, counts, buffer_size=len(z), max_D=len(d_len), seed=11,
                   flags=g.GPULDA_FLAG_LOGLIK) as s:
        s.corpus_load(z.copy(), w, d_len)
        z_buf = z.copy()
        for it in range(2):
            s.corpus_sweep(1)
            ch.sample_phi()
            r = ch.sweep(w, z_orc, d_len, want_ll=True)
            assert (s.corpus_z() == z_orc).all(), f"iteration {it}"
            assert (s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"] == ch.n).all()
            assert s.counters()["tokens"] == len(z) and s.counters()["docs"] == len(d_len)
            c = s.counters()
            assert c["sparse_work"] == int(r["stats"][2]) and c["sparse_draws"] == int(r["stats"][3])
            ll, _ = s.loglik()
            assert abs(ll - r["ll"]) <= 1e-4 * abs(r["ll"])
    with g.Sampler(0.05, 0.01, K, counts, buffer_size=len(z), max_D=len(d_len), seed=11) as s:
        k_d = np.zeros(len(d_len), np.uint32)
        for _ in range(2):
            s.sample_phi()
            s.sweep_buffer(0, z_buf, w, d_len, k_d)
    assert (z_buf == z_orc).all()
