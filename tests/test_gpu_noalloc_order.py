"""The allocation-free sweep of many documents, which finds their offsets and
their order on the device, against the resident sweep, bit for bit: numbers of
documents around the change from one way to the other and around its blocks of
4096 documents, and lengths around the steps of its bins, none and very long."""
import numpy as np
import pytest
import torch

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 3, 31, 32, 33, 60]


@pytest.mark.parametrize("long", [[], [511, 512, 513, 639, 640, 641, 20000, 65535]])
@pytest.mark.parametrize("K", [20, 700, 2500])
@pytest.mark.parametrize("n_docs", [2368, 2369, 4095, 4096, 4097, 12289])
def test_noalloc_sweep_of_many_documents(gpu_lib, n_docs, K, long):
    rng = np.random.default_rng(n_docs + K)
    V = 50
    d_len = rng.choice(LENGTHS, n_docs).astype(np.uint32)
    d_len[rng.permutation(n_docs)[:len(long)]] = long
    N = int(d_len.sum())
    w = rng.integers(0, V, N).astype(np.uint32)
    z = rng.integers(0, K, N).astype(np.uint32)
    counts = np.bincount(w, minlength=V).astype(np.uint32)
    with g.Sampler(0.1, 0.01, K, counts, buffer_size=16, max_D=4, seed=5) as s:
        s.corpus_load(z.copy(), w, d_len)
        s.corpus_sweep(1)
        want = s.corpus_z()
        n_want = s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"]
    dz, dw, dd = (torch.from_numpy(a.view(np.int32)).cuda() for a in (z, w, d_len))
    torch.cuda.synchronize()
    with g.Sampler(0.1, 0.01, K, counts, buffer_size=16, max_D=4, seed=5) as s:
        s.sample_phi()
        rc = g.lib().gpulda_sample_z_device_noalloc(dz.data_ptr(), dw.data_ptr(), dd.data_ptr(), n_docs, N, None)
        assert rc == g.GPULDA_OK
        torch.cuda.synchronize()
        got = dz.cpu().numpy().view(np.uint32)
        n = s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"]
    assert (got == want).all(), f"{(got != want).sum()} topics differ"
    assert (n == n_want).all()
