"""The give-up path of each tcgen05 kernel, exercised without faulting, trapping or hanging anything (see test_gpu_wait_limit.py): the limit is 2 ms,
and a test hook announces activations to their barrier without copying all of them.  The launch returns by itself, its status says so,
and a call enqueued right behind it, whose CTAs take over the shared and tensor memory that it leaves, is correct to the bit."""
import ctypes

import pytest
import torch

import kiln_b200
from kiln_b200 import _lib

pytestmark = pytest.mark.gpu


def _inputs(dev, m, k, n, groupsize, rank):
    gen = torch.Generator(device=dev)
    gen.manual_seed(m + k + n)
    words = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 16, 2 * n), dtype=torch.int32, device=dev, generator=gen)
    scales = (0.01 * torch.rand((1 if groupsize == -1 else k // 128, n), device=dev, generator=gen) + 1e-3).to(torch.float16)
    x = torch.randn((m, k), device=dev, generator=gen).to(torch.bfloat16)
    adapter = [torch.randn(s, device=dev, generator=gen).to(torch.bfloat16) for s in ((rank, k), (n, rank))] if rank else None
    return x, kiln_b200.MarlinPackedProj(words, scales, groupsize, k, n), adapter


def _give_up(call, drop, codes, limit_ns=2_000_000):
    lib = _lib.lib()
    want = call()
    torch.cuda.synchronize()
    assert lib.kiln_w4a16_check_device_status(None, None) == 0
    try:
        lib.kiln_w4a16_set_wait_limit_ns(limit_ns)
        lib.kiln_w4a16_test_drop_activation_load(drop)
        lost = call()
    finally:
        lib.kiln_w4a16_test_drop_activation_load(-1)
        lib.kiln_w4a16_set_wait_limit_ns(0)
    got = call()
    torch.cuda.synchronize()
    detail = ctypes.c_uint32(0)
    assert lib.kiln_w4a16_check_device_status(None, ctypes.byref(detail)) == _lib.ERR_TIMEOUT
    assert detail.value & 0xF00 in codes, hex(detail.value)
    assert lib.kiln_w4a16_check_device_status(None, None) == 0  # read and cleared
    assert torch.equal(got, want)
    assert lost.shape == want.shape


SMALL_BATCH = (0xA00, 0xB00, 0xD00, 0xE00, 0xF00)  # its waits: loads, issuers, results and the exchange, dequant, sums


# K splits: none, several, uneven ones, some with the receive buffer over the rings; K of a single stage and of more than the rings hold; an
# adapter's extra stage, which is not short; per-column scales
@pytest.mark.parametrize("m,k,n,groupsize,rank,splits", [
    (64, 1024, 256, 128, 0, 1), (17, 2560, 512, 128, 0, 1), (9, 128, 256, 128, 0, 1), (64, 2560, 4096, 128, 0, 4), (64, 640, 1024, 128, 0, 2),
    (100, 640, 1024, 128, 0, 2), (128, 9216, 2560, 128, 0, 6), (37, 2560, 2560, 128, 64, 3), (64, 128, 512, 128, 64, 1), (100, 4096, 2560, -1, 0, 3)])
def test_small_batch_kernel(cuda_device, m, k, n, groupsize, rank, splits):
    x, proj, adapter = _inputs(cuda_device, m, k, n, groupsize, rank)
    lib = _lib.lib()
    lib.kiln_w4a16_set_prefill_min_m(1)
    lib.kiln_w4a16_set_prefill_override(128, splits, 1, 0)
    try:
        _give_up(lambda: kiln_b200.matmul_bf16_lora(x, proj, *adapter, 0.5) if rank else kiln_b200.matmul_bf16(x, proj), 0, SMALL_BATCH)
    finally:
        lib.kiln_w4a16_set_prefill_override(0, 0, 0, 0)
        lib.kiln_w4a16_set_prefill_min_m(0)


@pytest.mark.parametrize("m,k,n,rank,swiglu", [(13, 2560, 512, 0, False), (16, 9216, 2560, 0, False), (13, 2560, 512, 64, False), (16, 2560, 512, 0, True),
                                               (64, 1152, 512, 0, False), (9, 128, 256, 0, False)])
def test_small_batch_kernel_with_fp32_scales(cuda_device, m, k, n, rank, swiglu):
    x, proj, adapter = _inputs(cuda_device, m, k, n, 128, rank)
    call = (lambda: kiln_b200.swiglu_gate_up(x, proj)) if swiglu else \
        (lambda: kiln_b200.matmul_bf16_lora(x, proj, *adapter, 0.5) if rank else kiln_b200.matmul_bf16(x, proj))
    _give_up(call, 0, SMALL_BATCH)


@pytest.mark.parametrize("bn,m,splits", [(128, 300, 1), (256, 300, 1), (128, 300, 2)])
def test_kernel_of_single_ctas(cuda_device, bn, m, splits):
    x, proj, _ = _inputs(cuda_device, m, 1024, 512, 128, 0)
    lib = _lib.lib()
    lib.kiln_w4a16_set_prefill_min_m(1)
    lib.kiln_w4a16_set_prefill_override(bn, splits, 1, 0)
    try:
        _give_up(lambda: kiln_b200.matmul_bf16(x, proj), 1, (0x100, 0x200, 0x300, 0x500, 0x600))
    finally:
        lib.kiln_w4a16_set_prefill_override(0, 0, 0, 0)
        lib.kiln_w4a16_set_prefill_min_m(0)


# both widths of tiles; K splits and stream-K, whose later passes run on what there is; several tiles per pair; an adapter, SwiGLU, per-column
# scales; a K shorter than the ring of stages
@pytest.mark.parametrize("bn,m,k,n,groupsize,rank,swiglu,splits,stream_k", [
    (128, 300, 1024, 512, 128, 0, False, 1, 0), (256, 300, 1024, 512, 128, 0, False, 1, 0), (256, 512, 2560, 2560, 128, 0, False, 3, 0),
    (256, 1000, 2560, 2560, 128, 0, False, 1, 1), (128, 4300, 256, 4096, 128, 0, False, 1, 0), (256, 300, 640, 1024, 128, 64, False, 1, 0),
    (256, 300, 640, 1024, 128, 0, True, 1, 0), (128, 300, 640, 512, -1, 0, False, 1, 0)])
def test_kernel_of_cta_pairs(cuda_device, bn, m, k, n, groupsize, rank, swiglu, splits, stream_k):
    x, proj, adapter = _inputs(cuda_device, m, k, n, groupsize, rank)
    call = (lambda: kiln_b200.swiglu_gate_up(x, proj)) if swiglu else \
        (lambda: kiln_b200.matmul_bf16_lora(x, proj, *adapter, 0.5) if rank else kiln_b200.matmul_bf16(x, proj))
    lib = _lib.lib()
    lib.kiln_w4a16_set_prefill_min_m(1)
    lib.kiln_w4a16_set_prefill_override(bn, splits, 2, stream_k)
    try:
        _give_up(call, 0, (0x100, 0x200, 0x300, 0x500, 0x600, 0x800, 0x900))
    finally:
        lib.kiln_w4a16_set_prefill_override(0, 0, 0, 0)
        lib.kiln_w4a16_set_prefill_min_m(0)


# clusters of 2, 5 and 8 CTAs (K = 512 each), one row tile and three, with the fp32 projection and with the bf16 one; a limit so short that
# only the least time that a CTA stays for its peers lets them finish
@pytest.mark.parametrize("m,k,rank,limit_ns", [(9, 1024, 16, 2_000_000), (16, 2560, 64, 2_000_000), (40, 4096, 64, 2_000_000), (100, 4096, 24, 2_000_000),
                                               (40, 4096, 64, 100_000)])
def test_exchange_of_the_lora_projection(cuda_device, m, k, rank, limit_ns):
    x, proj, adapter = _inputs(cuda_device, m, k, 2048, 128, rank)
    _give_up(lambda: kiln_b200.matmul_bf16_lora(x, proj, *adapter, 0.5), -2, (0xC00,), limit_ns)
