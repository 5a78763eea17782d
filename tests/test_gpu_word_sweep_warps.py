"""Above K = 1600 two blocks of eight warps, four documents each, do not fit an
SM's shared memory; smaller blocks then keep at least 12 of the 16 warps resident,
so a sweep over short lists takes at most 16/12 of what it takes at K = 1600."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


def _sweep_ms(K):
    """z sweep of 30,000 documents of 100 tokens over lists of 100 topics."""
    rng = np.random.default_rng(1)
    V, D, L = 4000, 30000, 100
    n0 = np.zeros((V, K), np.uint32)
    for w in range(V):
        n0[w, rng.permutation(1600)[:100]] = 40
    w = rng.integers(0, V, D * L).astype(np.uint32)
    z = rng.integers(0, 1600, D * L).astype(np.uint32)
    best = 1e9
    with g.Sampler(0.05, 0.0, K, np.bincount(w, minlength=V).astype(np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        for _ in range(6):
            s.write_counts(n0.reshape(-1))
            s.corpus_load(z, w, np.full(D, L, np.uint32))
            s.corpus_sweep(1)
            best = min(best, s.kernel_times()["z_sweep"])
    return best


@pytest.mark.parametrize("K", [1700, 1850, 2048])
def test_resident_warps_at_the_largest_dense_counts(gpu_lib, K):
    base, ms = _sweep_ms(1600), _sweep_ms(K)
    print(K, base, ms)
    assert ms < base * 16 / 12, f"{ms:.3f} ms at K={K}, {base:.3f} at K=1600"
