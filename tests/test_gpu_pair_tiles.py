"""GPU parity of the CTA-pair kernel with each of its tilings, forced through the tuning hook: 256- and 128-column tiles, K splits,
stream-K, ragged rows around a pair's 256 and a CTA's 128, per-column scales, LoRA.  <= 1e-2 against the fp64 oracle."""
import numpy as np
import pytest
import torch

import kiln_b200
import oracle
from kiln_b200 import _lib
from tests.test_gpu_epilogue import _lora, _proj
from tests.util import REL_TOL, from_torch_bf16, make_case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [256, 128])
@pytest.mark.parametrize("m,k,n,groupsize,splits,stream_k,rank", [
    (129, 128, 256, 128, 1, 0, 0), (255, 640, 512, 128, 1, 0, 0), (257, 1152, 768, 128, 2, 0, 0), (385, 2560, 1280, 128, 3, 0, 0),
    (512, 512, 9728, 128, 1, 1, 0), (1000, 9216, 2560, 128, 1, 1, 0), (300, 640, 512, -1, 1, 0, 0), (300, 1024, 2560, -1, 2, 0, 0),
    (4300, 256, 512, 128, 1, 0, 0), (300, 640, 1024, 128, 1, 0, 64), (300, 1024, 1280, 128, 2, 0, 16)])
def test_forced_pair_tiling_matches_the_oracle(cuda_device, bn, m, k, n, groupsize, splits, stream_k, rank):
    lib = _lib.lib()
    case = make_case(m, k, n, seed=m + n, groupsize=groupsize, device=cuda_device)
    ref = case["ref"].astype(np.float64)
    buf = torch.full((m + 2, n), 3.0, dtype=torch.bfloat16, device=cuda_device)
    lib.kiln_w4a16_set_prefill_min_m(1)
    lib.kiln_w4a16_set_prefill_override(bn, splits, 2, stream_k)
    try:
        if rank:
            la, lb = _lora(np.random.default_rng(m), rank, k, n)
            f = lambda bits: oracle.bf16_bits_to_f32(bits).astype(np.float64)
            ref = ref + (f(case["a"]) @ f(la).T) @ f(lb).T * 1.5
            bits = lambda b: torch.from_numpy(b.view(np.int16).copy()).view(torch.bfloat16).to(cuda_device)
            out = kiln_b200.matmul_bf16_lora(case["a_t"], _proj(case["q"], case["s"], groupsize, cuda_device), bits(la), bits(lb), 1.5)
        else:
            out = kiln_b200.marlin_w4a16_gemm(case["a_t"], case["b_t"], case["s_t"], groupsize, out=buf[1:m + 1])
        torch.cuda.synchronize()
    finally:
        lib.kiln_w4a16_set_prefill_override(0, 0, 0, 0)
        lib.kiln_w4a16_set_prefill_min_m(0)
    assert lib.kiln_w4a16_check_device_status(None, None) == 0
    assert rel_err(from_torch_bf16(out), ref.astype(np.float32)) <= REL_TOL
    assert (buf[0] == 3.0).all() and (buf[m + 1] == 3.0).all()
