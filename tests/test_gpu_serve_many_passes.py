"""Fold-in over the words' lists with more passes than one run of chunk numbers
holds (65,536 chunks) against the CPU oracle: the topics after a run's end are
those that it left, for requests of one chunk and of several.  (Chunk numbers
once covered all passes and wrapped at 2^32, which takes hours to reach.)"""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g
from gpupolyaurnlda_b200.serve import Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["launch", "persistent"])
@pytest.mark.parametrize("n_iter", [65535, 65536, 65537, 66001])
def test_many_passes(gpu_lib, oracle_lib, n_iter, mode):
    rng = np.random.default_rng(n_iter)
    K, V = 40, 12
    n0 = (rng.integers(1, 200, (V, K)) * (rng.random((V, K)) < 0.4)).astype(np.uint32)
    with g.Sampler(0.1, 0.0, K, np.full(V, 5, np.uint32), buffer_size=16, max_D=4, seed=2) as s:
        s.write_counts(n0.reshape(-1))
        s.sample_phi()
        st = s.read_state(n=False, S=False)
        srv = Server(n_iter, mode=mode, slots=2, seed=9, chain=3, pool_bytes=1 << 24)
    lengths = np.array([0, 1, 5, 32, 33], np.uint32)
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
