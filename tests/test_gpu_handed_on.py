"""Documents that outgrow the large-K sweep's register lists at their first
token, against the CPU oracle, bit for bit: the entry that the first token
leaves, which all lanes read for its gather, holds that token alone or most of
the document; first tokens in every position of a 32-entry group."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alone", [True, False])
def test_first_token_of_a_handed_on_document(gpu_lib, oracle_lib, alone):
    K, V, D, L = 4096, 64, 40, 700
    rng = np.random.default_rng(K + alone)
    z = np.stack([rng.permutation(K)[:L] for _ in range(D)])
    z.sort(axis=1)
    for d in range(D):  # the first token's topic: the document's d-th
        z[d, [0, d]] = z[d, [d, 0]]
        if not alone:
            z[d, 600:] = z[d, 0]
    z = z.reshape(-1).astype(np.uint32)
    w = rng.integers(0, V, D * L).astype(np.uint32)
    d_len = np.full(D, L, np.uint32)
    counts = np.bincount(w, minlength=V).astype(np.uint32)
    ch = oracle_lib.Chain(K, 0.05, 0.01, counts, seed=3)
    want = z.copy()
    with g.Sampler(0.05, 0.01, K, counts, buffer_size=16, max_D=4, seed=3) as s:
        s.corpus_load(z.copy(), w, d_len)
        for it in range(2):
            s.corpus_sweep(1)
            ch.sample_phi()
            ch.sweep(w, want, d_len)
            assert (s.corpus_z() == want).all(), f"iteration {it}"
            assert (s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"] == ch.n).all()
