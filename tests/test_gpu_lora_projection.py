"""GPU parity of the LoRA projection's kernels at the edges of their ranges (rows 8 / 9, the large tiles from 1025 rows of a rank above
32, ragged tiles of rows and of adapter rows, K splits of one to eight CTAs), through a GEMM with the delta, <= 1e-2 against fp64."""
import numpy as np
import pytest
import torch

import kiln_b200
import oracle
from oracle import C
from tests.test_gpu_epilogue import _lora, _proj
from tests.util import REL_TOL, from_torch_bf16, rel_err, to_torch_bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,r", [(8, 640, 512, 24), (9, 640, 512, 24), (65, 9216, 256, 64), (1024, 128, 512, 40), (1025, 128, 512, 40),
                                     (1025, 640, 512, 32), (1200, 2560, 256, 128), (2100, 256, 256, 72)])
def test_lora_delta_matches_the_oracle(cuda_device, m, k, n, r):
    a, q, s = oracle.synth_inputs(m, k, n, seed=m + r)
    la, lb = _lora(np.random.default_rng(m), r, k, n)
    f = lambda bits: oracle.bf16_bits_to_f32(bits).astype(np.float64)
    delta = (f(a) @ f(la).T) @ f(lb).T * 2.0
    base = C.gemm_fp64(a, q, s, 128).astype(np.float64)
    assert np.abs(delta).max() > 0.02 * np.abs(base).max()
    out = kiln_b200.matmul_bf16_lora(to_torch_bf16(a, cuda_device), _proj(q, s, 128, cuda_device), to_torch_bf16(la, cuda_device),
                                     to_torch_bf16(lb, cuda_device), 2.0)
    torch.cuda.synchronize()
    assert rel_err(from_torch_bf16(out), (base + delta).astype(np.float32)) <= REL_TOL
