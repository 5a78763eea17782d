"""The large-K sweep up to the largest K against the CPU oracle, bit for bit:
lists in shared memory with and without room for their q values (the change is
at K = 16,936), documents that stay in registers, pass 512 topics and hold up to
20,000, through the allocation-free call (whose lists are sized by K alone) and
the resident corpus (by its longest document)."""
import numpy as np
import pytest
import torch

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


def _corpus(K, lengths, V=24):
    rng = np.random.default_rng(K)
    z = np.concatenate([rng.permutation(K)[:L] if L <= K else rng.integers(0, K, L) for L in lengths])
    w = rng.integers(0, V, len(z))
    return z.astype(np.uint32), w.astype(np.uint32), np.array(lengths, np.uint32), \
        np.bincount(w, minlength=V).astype(np.uint32)


@pytest.mark.parametrize("lengths", [[1, 40, 300], [1, 40, 513, 2000, 700]])
@pytest.mark.parametrize("K", [2049, 16936, 16937, 20000, 32768])
def test_allocation_free_sweep(gpu_lib, oracle_lib, K, lengths):
    z, w, d_len, counts = _corpus(K, lengths)
    ch = oracle_lib.Chain(K, 0.05, 0.01, counts, seed=2)
    want = z.copy()
    dz, dw, dd = (torch.from_numpy(a.view(np.int32)).cuda() for a in (z, w, d_len))
    torch.cuda.synchronize()
    with g.Sampler(0.05, 0.01, K, counts, buffer_size=16, max_D=4, seed=2, flags=g.GPULDA_FLAG_LOGLIK) as s:
        for it in range(2):
            s.sample_phi()
            assert g.lib().gpulda_sample_z_device_noalloc(dz.data_ptr(), dw.data_ptr(), dd.data_ptr(), len(d_len),
                                                          len(z), None) == g.GPULDA_OK
            torch.cuda.synchronize()
            ch.sample_phi()
            r = ch.sweep(w, want, d_len, want_ll=True)
            assert (dz.cpu().numpy().view(np.uint32) == want).all(), f"iteration {it}"
            assert (s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"] == ch.n).all()
            c = s.counters()
            assert c["sparse_work"] == int(r["stats"][2]) and c["sparse_draws"] == int(r["stats"][3])
            assert abs(s.loglik()[0] - r["ll"]) <= 1e-4 * abs(r["ll"])


@pytest.mark.parametrize("K,lengths", [(16936, [16936, 600, 20]), (16937, [16937, 600, 20]), (20000, [17000, 600, 20]),
                                       (32768, [20000, 16904, 3])])
def test_resident_corpus_with_a_document_of_most_topics(gpu_lib, oracle_lib, K, lengths):
    z, w, d_len, counts = _corpus(K, lengths)
    ch = oracle_lib.Chain(K, 0.05, 0.01, counts, seed=4)
    want = z.copy()
    with g.Sampler(0.05, 0.01, K, counts, buffer_size=16, max_D=4, seed=4) as s:
        s.corpus_load(z.copy(), w, d_len)
        for it in range(2):
            s.corpus_sweep(1)
            ch.sample_phi()
            ch.sweep(w, want, d_len)
            assert (s.corpus_z() == want).all(), f"iteration {it}"
            assert (s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"] == ch.n).all()
