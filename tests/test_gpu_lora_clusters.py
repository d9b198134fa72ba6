"""The LoRA projection for every cluster size (K = 512 d gives d CTAs), also those that do not divide a tile, rows of one tile and of two, and
ranks that fill a column tile or not.  The base weight is tiny, so the result is the delta: tolerance 1e-2 of the largest, as elsewhere."""
import pytest
import torch

import kiln_b200
from kiln_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [8, 24, 64])
@pytest.mark.parametrize("k", [128, 512, 1024, 1536, 2048, 2560, 3072, 3584, 4096])
def test_projection(cuda_device, k, r):
    _check(cuda_device, k, r, (1, 4, 8, 17, 40, 130))


def _check(cuda_device, k, r, rows):
    n, gen = 256, torch.Generator(device=cuda_device).manual_seed(k + r)
    w = torch.full((k // 16, 2 * n), -0x77777778, dtype=torch.int32, device=cuda_device)  # every weight (8 - 8) s = 0
    proj = kiln_b200.MarlinPackedProj(w, torch.full((k // 128, n), 0.01, dtype=torch.float16, device=cuda_device), 128, k, n)
    for m in rows:
        x = torch.randn((m, k), device=cuda_device, generator=gen).bfloat16()
        a = torch.randn((r, k), device=cuda_device, generator=gen).bfloat16()
        b = torch.randn((n, r), device=cuda_device, generator=gen).bfloat16()
        out = kiln_b200.matmul_bf16_lora(x, proj, a, b, 0.5)
        torch.cuda.synchronize()
        assert _lib.lib().kiln_w4a16_check_device_status(None, None) == 0
        ref = 0.5 * (x.double() @ a.double().T) @ b.double().T
        assert float((out.double() - ref).abs().max() / ref.abs().max()) <= 1e-2, m


# the line between dot products and tiles: four rows, rows x rank of 128, K of 1280; ranks that are no multiple of a block's eight warps x rows
@pytest.mark.parametrize("k,r,rows", [(128, 8, (1, 4, 5)), (1280, 32, (1, 2, 4, 5)), (1280, 40, (3, 4)), (1408, 32, (4,)), (640, 128, (1, 2)), (1024, 120, (1,))])
def test_few_rows_of_a_short_k(cuda_device, k, r, rows):
    _check(cuda_device, k, r, rows)


# large tiles: clusters of 1 to 8 CTAs, shares that are no multiple of the threads, and counts of tiles for which clusters of eight do not fit at once
@pytest.mark.parametrize("m,k,r", [(1100, 128, 64), (2100, 512, 128), (1100, 256, 72), (3000, 512, 64), (1100, 384, 64), (2100, 512, 40), (1100, 512, 64),
                                   (16384, 128, 40)])
def test_large_tiles(cuda_device, m, k, r):
    _check(cuda_device, k, r, (m,))
