"""Grouped launches of the small-batch kernel and of its variant with fp32 scales, against the fp64 oracle, and their number of launches.
Tolerance: max|out - ref| / max|ref| <= 1e-2, as for single launches."""
import numpy as np
import pytest
import torch

import kiln_b200
from kiln_b200 import _lib
import oracle
from oracle import C
from tests.util import REL_TOL, from_torch_bf16, rel_err, to_torch_bf16

pytestmark = pytest.mark.gpu


# (rows, K, columns of each, group size, launches): nine to 32 rows in one launch; above, neighbours of one kind; five problems, the decode kernel
# or, for more rows of a long K, two launches; rows that are no multiple of four, and several CTAs of 16 rows; group sizes -1; the 128-row
# variant; one K stage; decode up to 8 rows; either side of the lines between the decode kernel and the variant that the columns of all draw:
# half the GPU's tiles up to 8 rows, a second wave of CTAs, split or not
@pytest.mark.parametrize("m,k,ns,groupsize,launches", [
    (9, 640, (512, 256, 256), 128, 1), (16, 2560, (4096, 512, 512), 128, 1), (29, 640, (4096, 512, 512), 128, 1), (13, 384, (256,) * 5, 128, 1), (17, 5248, (256,) * 5, 128, 2),
    (13, 640, (512, 256), -1, 1), (37, 640, (4096, 512, 512), 128, 2), (50, 640, (512, 4096, 2048, 512), 128, 3), (101, 1280, (2048, 4096), 128, 1),
    (64, 2560, (2048, 2048, 2048), 128, 1), (128, 128, (1280, 1280), 128, 1), (77, 640, (2048, 2048), -1, 1), (8, 640, (512, 256), 128, 1),
    (7, 256, (4864, 4608), 128, 1), (7, 256, (4864, 4864), 128, 1), (4, 1024, (3072, 1024), 128, 1), (16, 256, (9472, 9728), 128, 1),
    (17, 640, (4864, 4608), 128, 1), (17, 640, (4864, 4864), 128, 1), (17, 2560, (4864, 4864), 128, 1), (13, 5248, (3328, 6400), 128, 1),
    (12, 5248, (3328, 6400), 128, 1)])
def test_alike_problems_share_a_launch(cuda_device, m, k, ns, groupsize, launches):
    xs, projs, refs = [], [], []
    for i, n in enumerate(ns):
        a, q, s = oracle.synth_inputs(m, k, n, seed=m + n + i, groupsize=groupsize)
        packed, sp = kiln_b200.pack.repack(q, s, groupsize)
        projs.append(kiln_b200.MarlinPackedProj(torch.from_numpy(packed).to(cuda_device),
                                                torch.from_numpy(sp.view(np.int16).copy()).view(torch.float16).to(cuda_device), groupsize, k, n))
        xs.append(to_torch_bf16(a, cuda_device))
        refs.append(C.gemm_fp64(a, q, s, groupsize))
    lib = _lib.lib()
    before = lib.kiln_w4a16_launch_count()
    outs = kiln_b200.grouped_matmul_bf16(xs, projs)
    torch.cuda.synchronize()
    assert lib.kiln_w4a16_check_device_status(None, None) == 0
    assert lib.kiln_w4a16_launch_count() - before == launches
    for out, ref in zip(outs, refs):
        assert rel_err(from_torch_bf16(out), ref) <= REL_TOL


# K of 112 and 128 stages, where a CTA takes at most 96 and each problem by itself has two splits or more: the columns of all of them ask for fewer
@pytest.mark.parametrize("m,k,ns,launches", [(16, 14336, (7168, 7168), 1), (64, 16384, (9216, 9216), 1), (100, 16384, (8192, 1024, 1024), 2),
                                             (13, 28672, (4096, 1024, 1024), 1)])
def test_alike_problems_of_a_long_k(cuda_device, m, k, ns, launches):
    gen = torch.Generator(device=cuda_device).manual_seed(m + k)
    xs, projs, refs = [], [], []
    for n in ns:
        q = torch.randint(0, 16, (k, n), dtype=torch.uint8, device=cuda_device, generator=gen)
        s = (0.01 * torch.rand((k // 128, n), device=cuda_device, generator=gen) + 1e-3).half()
        packed, sp = kiln_b200.pack.repack(q.cpu().numpy(), s.cpu().numpy(), 128)
        projs.append(kiln_b200.MarlinPackedProj(torch.from_numpy(packed).to(cuda_device),
                                                torch.from_numpy(sp.view(np.int16).copy()).view(torch.float16).to(cuda_device), 128, k, n))
        xs.append(torch.randn((m, k), device=cuda_device, generator=gen).bfloat16())
        w = (q.view(k // 128, 128, n).double() - 8.0) * s.double()[:, None]
        refs.append((xs[-1].double() @ w.view(k, n)).float().cpu().numpy())
    lib = _lib.lib()
    before = lib.kiln_w4a16_launch_count()
    outs = kiln_b200.grouped_matmul_bf16(xs, projs)
    torch.cuda.synchronize()
    assert lib.kiln_w4a16_check_device_status(None, None) == 0
    assert lib.kiln_w4a16_launch_count() - before == launches
    for out, ref in zip(outs, refs):
        assert rel_err(from_torch_bf16(out), ref) <= REL_TOL
