"""The large-K sweep with a bit for each of a word's topics, which models whose
Phi does not fit the cache and sweeps of many documents use, against the same
documents in small sweeps without them, bit for bit: ragged numbers of topics,
lists of every number of entries a lane and some handed on, words of no, few
and most topics."""
import numpy as np
import pytest

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, g.GPULDA_FLAG_LOGLIK])
@pytest.mark.parametrize("K", [2049, 2500, 4111])
def test_bits_change_no_topic(gpu_lib, K, flags):
    rng = np.random.default_rng(K)
    V = (600 << 20) // (4 * K)  # Phi of 600 MB
    used = rng.permutation(V)[:300]
    d_len = np.concatenate([rng.integers(0, 12, 24000), [31, 32, 33, 64, 65, 96, 127, 128, 129, 190, 250, 400, 700, 1500]])
    d_len = rng.permutation(d_len).astype(np.uint32)
    N = int(d_len.sum())
    w = used[np.minimum(rng.geometric(0.02, N) - 1, 299)].astype(np.uint32)
    z = rng.integers(0, K, N).astype(np.uint32)
    counts = np.bincount(w, minlength=V).astype(np.uint32)
    out = []
    for pieces in (1, 3):
        with g.Sampler(0.05, 0.01, K, counts, buffer_size=N, max_D=len(d_len), seed=3, flags=flags) as s:
            zz = z.copy()
            for _ in range(2):
                s.sample_phi()
                cut = [len(d_len) * p // pieces for p in range(pieces + 1)]
                for d0, d1 in zip(cut, cut[1:]):
                    t0, t1 = int(d_len[:d0].sum()), int(d_len[:d1].sum())
                    zp = zz[t0:t1].copy()
                    s.sweep_buffer(0, zp, w[t0:t1].copy(), d_len[d0:d1].copy(), np.zeros(d1 - d0, np.uint32))
                    zz[t0:t1] = zp
            out.append((zz, s.read_state(q=False, alias=False, A=False, S=False, nnz=False)["n"],
                        s.loglik()[0] if flags else 0.0))
    assert (out[0][0] == out[1][0]).all(), f"{(out[0][0] != out[1][0]).sum()} topics differ"
    assert (out[0][1] == out[1][1]).all()
    assert abs(out[0][2] - out[1][2]) <= 1e-4 * abs(out[1][2])
