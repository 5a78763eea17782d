"""A large-K model whose sweeps use the hash map keeps no words' bits, which
those sweeps do not read (20 MB here, written by every alias build)."""
import numpy as np
import pytest
import torch

import gpupolyaurnlda_b200 as g

pytestmark = pytest.mark.gpu


def _model_bytes(flags):
    K, V = 4096, 40000  # q of 655 MB
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with g.Sampler(0.1, 0.01, K, np.full(V, 3, np.uint32), buffer_size=16, max_D=4, flags=flags):
        return before - torch.cuda.mem_get_info()[0]


def test_no_bits_beside_the_hash_map(gpu_lib):
    _model_bytes(0)  # loads what the process loads once
    assert _model_bytes(0) - _model_bytes(g.GPULDA_FLAG_HASHMAP) > 15 << 20
