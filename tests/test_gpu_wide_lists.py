"""Words of more topics than a warp of the alias build takes go to a block with
their draws listed, against the CPU oracle, bit for bit: the draw that is one too
many in each of the row's last cells (rows of odd length start at every offset
from 16 bytes), and listed draws of which one rounds to q = 0."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("huge_topic", [False, True])
@pytest.mark.parametrize("K", [257, 639, 1279, 1281, 2047, 2049, 4099])
def test_wide_lists_match_oracle(gpu_lib, oracle_lib, K, huge_topic):
    rng = np.random.default_rng(K)
    most = 256 if K <= 2048 else 512
    V = 24
    n0 = np.zeros((V, K), np.uint32)
    for w in range(V):  # (a Poisson draw of 40 or more is positive but for e^-40)
        last = K - 1 - w % min(6, K - most)
        n0[w, rng.permutation(last)[:most]] = rng.integers(40, 90, most)
        n0[w, last] = 50
        if w >= 12:  # more behind it
            n0[w, last + 1:] = 45
    if huge_topic:
        n0[:, 1] = rng.integers(1, 4, V)
        n0[0, 1] = 3000000000
        n0[13, 1] = 3000000000
    with g.Sampler(0.1, 0.0, K, np.full(V, 10, np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        s.write_counts(n0.reshape(-1))
        s.sample_phi()
        st = s.read_state()
    phi = oracle_lib.phi_step(K, V, 0.0, n0.reshape(-1).copy(), 0, 5, 0)
    st["alias"] = oracle_lib.live_alias_entries(st["alias"], st["nnz"], K)
    phi["alias"] = oracle_lib.live_alias_entries(phi["alias"], phi["nnz"], K)
    assert (phi["nnz"] >= most).all() and (phi["nnz"] > most).any(), "the lists have other lengths than meant"
    for key in ("S", "q", "A", "nnz", "alias"):
        assert (st[key].reshape(-1) == phi[key].reshape(-1)).all(), key
