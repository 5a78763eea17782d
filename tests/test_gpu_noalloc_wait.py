"""The Phi step after an allocation-free sweep waits for everything that the
call queued on the caller's stream, also where a launch of it was refused: the
call comes behind 0.1 s of other work on that stream, and the Phi step (which
the host waits for) must not be over before it.  K around the largest list in
shared memory, where a refused launch is the nearest."""
import numpy as np
import pytest
import torch

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [100, 4096, 16936, 16937, 32768])
@pytest.mark.parametrize("n_docs", [3, 2500])
def test_phi_step_waits_for_the_call(gpu_lib, K, n_docs):
    V = 20
    rng = np.random.default_rng(K)
    d_len = np.full(n_docs, 3, np.uint32)
    N = int(d_len.sum())
    w = rng.integers(0, V, N).astype(np.uint32)
    z = rng.integers(0, K, N).astype(np.uint32)
    dz, dw, dd = (torch.from_numpy(a.view(np.int32)).cuda() for a in (z, w, d_len))
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    L = g.lib()
    with g.Sampler(0.1, 0.01, K, np.bincount(w, minlength=V).astype(np.uint32), buffer_size=16, max_D=4, seed=5) as s:
        for first in (True, False):  # (the first call may wait for the GPU while its kernels are loaded)
            s.sample_phi()
            if not first:
                with torch.cuda.stream(st):
                    torch.cuda._sleep(200_000_000)
            L.gpulda_sample_z_device_noalloc(dz.data_ptr(), dw.data_ptr(), dd.data_ptr(), n_docs, N, st.cuda_stream)
            L.gpulda_last_error()  # whether the call went through is not this test's
            assert first or not st.query(), "the other work was over too early for the test"
            s.sample_phi()
            assert st.query(), "the Phi step ran ahead of the sweep"
    torch.cuda.synchronize()
