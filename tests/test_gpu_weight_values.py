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
SHAPES = [(16, 2048), (48, 2048), (128, 2048), (129, 2048), (256, 18432), (300, 256)]


@pytest.mark.parametrize("groupsize", [128, -1])
@pytest.mark.parametrize("m,n", SHAPES)
def test_a_weight_comes_out_as_it_was_packed(cuda_device, m, n, groupsize):
    _check(cuda_device, m, n, groupsize, 1.0, rng_scales=lambda rng: np.concatenate(
        [[1, 2, 3, 0x3FF, 0x400, 0x7BFF, 0x7BFE, 0x3C00, 0x2E66], rng.integers(1, 0x7C00, 1024)]))


@pytest.mark.parametrize("groupsize", [128, -1])
@pytest.mark.parametrize("m,n", SHAPES)
def test_tiny_results_keep_their_bits(cuda_device, m, n, groupsize):
    """Activations of 2^-112, scales from 2^-6 to 2^4: results down to 2^-118, whose eight bits are still there at the weights' factor of 2^-22
    (the sums' last bit is 2^-149)."""
    _check(cuda_device, m, n, groupsize, 2.0 ** -112, rng_scales=lambda rng: rng.integers(0x2400, 0x4C00, 1024))


def _check(cuda_device, m, n, groupsize, hot_value, rng_scales):
    k = 256
    rng = np.random.default_rng(m + n)
    q = rng.integers(0, 16, (k, n), dtype=np.uint8)
    rows = 1 if groupsize == -1 else k // 128
    bits = np.resize(rng_scales(rng), rows * n)
    s = rng.permutation(bits).astype(np.uint16).view(np.float16).reshape(rows, n)
    packed, sp = kiln_b200.pack.repack(q, s, groupsize)
    hot = rng.integers(0, k, m)
    x = torch.zeros((m, k), dtype=torch.bfloat16, device=cuda_device)
    x[torch.arange(m, device=cuda_device), torch.from_numpy(hot).to(cuda_device)] = hot_value
    out = kiln_b200.marlin_w4a16_gemm(x, torch.from_numpy(packed).to(cuda_device),
                                      torch.from_numpy(sp.view(np.int16).copy()).view(torch.float16).to(cuda_device), groupsize)
    torch.cuda.synchronize()
    assert _lib.lib().kiln_w4a16_check_device_status(None, None) == 0
    scale = torch.from_numpy(s.astype(np.float32)[(np.zeros(m, dtype=int) if groupsize == -1 else hot // 128)])
    if m > 16 and groupsize == 128 and not (n <= 1024 and m <= 256):
        scale = scale.bfloat16().float()
    want = ((torch.from_numpy(q[hot].astype(np.float32)) - 8.0) * scale * hot_value).bfloat16()
    assert torch.equal(out.cpu(), want)
