"""The alias build, a word to a warp or to a block by its number of topics,
against the CPU oracle, bit for bit: words of every number of topics around the
change from one to the other and around a warp's steps, rows that start at
every offset from 16 bytes, and a topic so large that small draws round to
q = 0 and leave the list."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu

LISTS = [0, 1, 2, 3, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1000, 2048, 2049, 2500]


@pytest.mark.parametrize("huge_topic", [False, True])
@pytest.mark.parametrize("K", [1, 5, 31, 33, 255, 256, 257, 513, 1000, 2047, 2049, 2501])
def test_alias_rows_match_oracle(gpu_lib, oracle_lib, K, huge_topic):
    rng = np.random.default_rng(K)
    lists = [n for n in LISTS if n <= K] + [K]
    V = len(lists) + 40
    n0 = np.zeros((V, K), np.uint32)
    for w, n in enumerate(lists):  # (a Poisson draw of 40 or more is positive but for e^-40)
        n0[w, rng.permutation(K)[:n]] = rng.integers(40, 90, n)
    n0[len(lists):] = rng.integers(0, 3, (V - len(lists), K)) * (rng.random((V - len(lists), K)) < 0.1)
    if huge_topic:
        n0[len(lists):len(lists) + 2, 0] = 3000000000
        n0[len(lists) + 2:, 0] = 1
    with g.Sampler(0.1, 0.0, K, np.full(V, 10, np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        s.write_counts(n0.reshape(-1))
        s.sample_phi()
        st = s.read_state()
    phi = oracle_lib.phi_step(K, V, 0.0, n0.reshape(-1).copy(), 0, 5, 0)
    assert huge_topic or [int(x) for x in phi["nnz"][:len(lists)]] == lists, "the lists have other lengths than meant"
    st["alias"] = oracle_lib.live_alias_entries(st["alias"], st["nnz"], K)
    phi["alias"] = oracle_lib.live_alias_entries(phi["alias"], phi["nnz"], K)
    for key in ("S", "q", "A", "nnz", "alias"):
        assert (st[key].reshape(-1) == phi[key].reshape(-1)).all(), key
