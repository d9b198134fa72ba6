"""Single weights through the tcgen05 kernels: with one-hot activations a result IS a dequantised weight, so it must be
bf16((nibble - 8) * bf16(scale)) to the bit, for every nibble and scales from the smallest fp16 subnormal to the largest number; in the
variant that applies fp32 scales, bf16((nibble - 8) * scale)."""
import numpy as np
import pytest
import torch

import kiln_b200
from kiln_b200 import _lib

pytestmark = pytest.mark.gpu


# rows -> kernel: 16 fp32 scales; 48, 128 small-batch; 129, 256 CTA pairs (split K or whole tiles); 300 x 256 columns: single-CTA tiles
@pytest.mark.parametrize("groupsize", [128, -1])
@pytest.mark.parametrize("m,n", [(16, 2048), (48, 2048), (128, 2048), (129, 2048), (256, 18432), (300, 256)])
def test_a_weight_comes_out_as_it_was_packed(cuda_device, m, n, groupsize):
    k = 256
    rng = np.random.default_rng(m + n)
    q = rng.integers(0, 16, (k, n), dtype=np.uint8)
    rows = 1 if groupsize == -1 else k // 128
    bits = np.resize(np.concatenate([[1, 2, 3, 0x3FF, 0x400, 0x7BFF, 0x7BFE, 0x3C00, 0x2E66], rng.integers(1, 0x7C00, 1024)]), rows * n)
    s = rng.permutation(bits).astype(np.uint16).view(np.float16).reshape(rows, n)
    packed, sp = kiln_b200.pack.repack(q, s, groupsize)
    hot = rng.integers(0, k, m)
    x = torch.zeros((m, k), dtype=torch.bfloat16, device=cuda_device)
    x[torch.arange(m, device=cuda_device), torch.from_numpy(hot).to(cuda_device)] = 1.0
    out = kiln_b200.marlin_w4a16_gemm(x, torch.from_numpy(packed).to(cuda_device),
                                      torch.from_numpy(sp.view(np.int16).copy()).view(torch.float16).to(cuda_device), groupsize)
    torch.cuda.synchronize()
    assert _lib.lib().kiln_w4a16_check_device_status(None, None) == 0
    scale = torch.from_numpy(s.astype(np.float32)[(np.zeros(m, dtype=int) if groupsize == -1 else hot // 128)])
    if m > 16 and groupsize == 128 and not (n <= 1024 and m <= 256):
        scale = scale.bfloat16().float()
    want = ((torch.from_numpy(q[hot].astype(np.float32)) - 8.0) * scale).bfloat16()
    assert torch.equal(out.cpu(), want)
