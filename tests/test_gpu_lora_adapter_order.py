"""An adapter that the launch right before wrote: the projection starts while that launch still runs (programmatic dependent launch) and must
read the adapter after its end.  Results are compared with those of synchronised calls, bit for bit."""
import re
from pathlib import Path

import pytest
import torch

import kiln_b200


def test_no_load_of_the_projection_may_move_across_the_wait():
    """The compiler may move a read-only load (__ldg) up; the adapter and the activations are read by volatile assembly alone."""
    src = (Path(kiln_b200.__file__).parent / "csrc" / "epilogue_w4a16.cu").read_text()
    assert "__ldg" not in re.sub(r"//[^\n]*", "", src)


@pytest.mark.gpu
@pytest.mark.parametrize("m,r", [(4, 64), (40, 16), (130, 64), (1200, 64)])
def test_an_adapter_written_by_the_launch_before(cuda_device, m, r):
    k, n, gen = 2560, 2560, torch.Generator(device=cuda_device).manual_seed(m)
    words = lambda cols: torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 16, 2 * cols), dtype=torch.int32, device=cuda_device, generator=gen)
    scales = lambda cols: (1e-3 * torch.rand((k // 128, cols), device=cuda_device, generator=gen) + 1e-4).half()
    maker, proj = (kiln_b200.MarlinPackedProj(words(c), scales(c), 128, k, c) for c in (k, n))
    x = torch.randn((m, k), device=cuda_device, generator=gen).bfloat16()
    b = torch.randn((n, r), device=cuda_device, generator=gen).bfloat16()
    seeds = [torch.randn((r, k), device=cuda_device, generator=gen).bfloat16() for _ in range(2)]
    adapter = torch.empty((r, k), dtype=torch.bfloat16, device=cuda_device)
    make = lambda i: kiln_b200.marlin_w4a16_gemm(seeds[i], maker.b_packed, maker.scales, 128, out=adapter)
    want = []
    for i in range(2):
        make(i)
        torch.cuda.synchronize()
        want.append(kiln_b200.matmul_bf16_lora(x, proj, adapter, b, 0.5))
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    outs = []
    for i in range(40):
        make(i % 2)
        outs.append(kiln_b200.matmul_bf16_lora(x, proj, adapter, b, 0.5))
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out, want[i % 2]), i
