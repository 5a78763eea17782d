"""The Phi draw's mappings of rows to threads against the CPU oracle, bit for
bit: topics in every number of groups of four that changes how many rows a
block takes side by side, numbers of topics that are no multiple of four, few
and many words, counts on both sides of the inversion tables."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8, 20, 127, 128, 132, 333, 508, 512, 516, 1000, 1025, 1028, 2050])
@pytest.mark.parametrize("V", [1, 51, 1203])
def test_phi_step_matches_oracle(gpu_lib, oracle_lib, K, V):
    rng = np.random.default_rng(K * 7 + V)
    n0 = (rng.integers(0, 90, K * V) * (rng.random(K * V) < 0.4)).astype(np.uint32)
    with g.Sampler(0.1, 0.01, K, np.full(V, 5, np.uint32), buffer_size=16, max_D=4, seed=8) as s:
        s.write_counts(n0)
        s.sample_phi()
        st = s.read_state()
    ref = oracle_lib.phi_step(K, V, 0.01, n0.copy(), 0, 8, 0)
    assert (st["S"] == ref["S"]).all()
    assert (st["q"] == ref["q"]).all() and (st["A"] == ref["A"]).all() and (st["nnz"] == ref["nnz"]).all()
    assert not st["n"].any()
