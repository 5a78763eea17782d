"""Models, batches and servers that fit the free memory only without the words'
lists (a table that sweeps are faster with): they are built without, a later
allocation of the library's takes the lists' place, and results are the same bit
for bit."""
import numpy as np
import pytest
import torch

import gpupolyaurnlda_b200 as g
from gpupolyaurnlda_b200 import batch
from gpupolyaurnlda_b200.serve import Server

pytestmark = pytest.mark.gpu

MB = 1 << 20
K, V = 1000, 20000  # 24 bytes a cell: 480 MB; the words' lists: 174 MB


def _hold_all_but(n_bytes):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - n_bytes, dtype=torch.uint8, device="cuda")


def _documents(rng, N, K, V):
    L = 100
    return rng.integers(0, K, N).astype(np.uint32), rng.integers(0, V, N).astype(np.uint32), \
        np.full(N // L, L, np.uint32)


def _warm_up():
    """Loads the kernels, which takes memory of its own."""
    rng = np.random.default_rng(0)
    z, w, d = _documents(rng, 3000, 200, 50)
    with g.Sampler(0.1, 0.01, 200, np.bincount(w, minlength=50).astype(np.uint32), buffer_size=16, max_D=4) as s:
        s.corpus_load(z, w, d)
        s.corpus_sweep(2)


@pytest.mark.parametrize("when", ["model", "corpus"])
def test_chain(gpu_lib, oracle_lib, when):
    _warm_up()
    rng = np.random.default_rng(1)
    N = 200000 if when == "model" else 8000000
    z, w, d_len = _documents(rng, N, K, V)
    counts = np.bincount(w, minlength=V).astype(np.uint32)
    hold = _hold_all_but(580 * MB) if when == "model" else None
    try:
        s = g.Sampler(0.05, 0.01, K, counts, buffer_size=16, max_D=4, seed=3)
        try:
            if when == "corpus":  # 64 MB of tokens into 50: the lists make way
                hold = _hold_all_but(50 * MB)
            s.corpus_load(z.copy(), w, d_len)
            s.corpus_sweep(2)
            got = s.corpus_z()
        finally:
            s.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    ch = oracle_lib.Chain(K, 0.05, 0.01, counts, seed=3)
    for _ in range(2):
        ch.sample_phi()
        ch.sweep(w, z, d_len)
    assert (got == z).all(), f"{(got != z).sum()} topics differ"


@pytest.mark.parametrize("when", ["create", "tune"])
def test_batch(gpu_lib, when):
    rng = np.random.default_rng(2)
    problems = []
    for p in range(3):
        z, w, d_len = _documents(rng, 30000, 1000, 8000)
        problems.append(batch.ProblemSpec(0.05, 0.01, 1000, np.bincount(w, minlength=8000).astype(np.uint32), z, w, d_len,
                                          seed=p, loglik=False))
    with batch.BatchChains(problems) as chains:
        with_lists = chains.info()["device_bytes"]
        chains.sweep(2)
        want = [chains.z(p) for p in range(3)]
    # 24e6 cells: 576 MB, the lists 209 MB, the tuner's copy of the counts 96 MB
    hold = _hold_all_but(700 * MB) if when == "create" else None
    try:
        with batch.BatchChains(problems) as chains:
            if when == "tune":
                hold = _hold_all_but(60 * MB)
                assert chains.info()["device_bytes"] == with_lists
                chains.tune()
            assert chains.info()["device_bytes"] < with_lists - 200_000_000
            chains.sweep(2)
            got = [chains.z(p) for p in range(3)]
    finally:
        del hold
        torch.cuda.empty_cache()
    for a, b in zip(got, want):
        assert (a == b).all()


@pytest.mark.parametrize("mode", ["launch", "persistent"])
def test_server(gpu_lib, mode):
    rng = np.random.default_rng(3)
    q = (rng.integers(1, 1 << 26, (V, K)) * (rng.random((V, K)) < 0.02)).astype(np.uint32)
    lengths = np.array([1, 40, 300], np.uint32)
    words = rng.integers(0, V, int(lengths.sum())).astype(np.uint32)
    ids = np.arange(3, dtype=np.uint64)
    out = []
    for tight in (False, True):
        hold = _hold_all_but(480 * MB) if tight else None  # the model's 20 bytes a cell: 400 MB
        try:
            with Server(3, mode=mode, slots=2, q=q, K=K, alpha=0.05, seed=1, pool_bytes=16 * MB) as srv:
                srv.submit(ids, lengths, words)
                srv.drain()
                r = srv.poll(3)
                order = np.argsort(r["ids"])
                out.append((r["theta"][order], r["ll"][order]))
        finally:
            del hold
            torch.cuda.empty_cache()
    assert (out[0][0].view(np.uint32) == out[1][0].view(np.uint32)).all()
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-12)
