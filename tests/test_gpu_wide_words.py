"""Words of more topics than a warp of the alias build takes are built side by
side, a block to each: four such words take little longer than one (they once
waited for each other in one block, and took four times as long)."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


def _alias_ms(K, V):
    n0 = np.full(V * K, 50, np.uint32)
    with g.Sampler(0.1, 0.0, K, np.full(V, 10, np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        best = 1e9
        for _ in range(6):
            s.write_counts(n0)
            s.sample_phi()
            best = min(best, s.kernel_times()["alias_build"])
    return best


@pytest.mark.parametrize("K", [2000, 8000])
def test_wide_words_do_not_wait_for_each_other(gpu_lib, K):
    one, four = _alias_ms(K, 1), _alias_ms(K, 4)
    assert four < 2 * one, f"{four * 1e3:.0f} us for four words, {one * 1e3:.0f} for one"
