"""GPU parity of the small-batch kernel's variant that applies the group scales and a LoRA delta in fp32, which the built-in rule takes for
few rows or few columns.  Against the fp64 oracle (<= 1e-2), and no further from it than the decode kernel on the same inputs."""
import numpy as np
import pytest
import torch

import kiln_b200
import oracle
from kiln_b200 import _lib
from oracle import C
from tests.test_gpu_epilogue import _gate_up_case, _lora, _proj, _silu
from tests.util import REL_TOL, from_torch_bf16, rel_err, to_torch_bf16

pytestmark = pytest.mark.gpu


# rows: both sides of a block of 16, the last block with one row; K: fewer stages than teams, than slots, and more; K splits from
# one to eight; ranks that the splits share unevenly or not at all
@pytest.mark.parametrize("m,k,n,groupsize,rank", [
    (4, 128, 256, 128, 0), (8, 384, 8192, 128, 0), (9, 640, 1024, 128, 0), (16, 2560, 18432, 128, 0), (13, 9216, 2560, 128, 0),
    (15, 1152, 38400, 128, 0), (17, 2560, 512, 128, 0), (256, 2560, 1024, 128, 0), (255, 128, 256, 128, 0), (16, 4096, 2560, -1, 0),
    (33, 1024, 512, -1, 0), (3, 2560, 512, 128, 8), (5, 2560, 4096, 128, 16), (16, 128, 256, 128, 128), (24, 2560, 4096, 128, 64),
    (241, 640, 1024, 128, 40)])
def test_matches_the_oracle_and_the_decode_kernel(cuda_device, m, k, n, groupsize, rank):
    lib = _lib.lib()
    a, q, s = oracle.synth_inputs(m, k, n, seed=m + k + n, groupsize=groupsize)
    ref = C.gemm_fp64(a, q, s, groupsize).astype(np.float64)
    proj, x = _proj(q, s, groupsize, cuda_device), to_torch_bf16(a, cuda_device)
    buf = torch.full((m + 2, n), 3.0, dtype=torch.bfloat16, device=cuda_device)
    if rank:
        la, lb = _lora(np.random.default_rng(m), rank, k, n)
        f = lambda bits: oracle.bf16_bits_to_f32(bits).astype(np.float64)
        ref = ref + (f(a) @ f(la).T) @ f(lb).T * 1.5
        la, lb = to_torch_bf16(la, cuda_device), to_torch_bf16(lb, cuda_device)

    def run():
        if rank:
            return kiln_b200.matmul_bf16_lora(x, proj, la, lb, 1.5)
        return kiln_b200.marlin_w4a16_gemm(x, proj.b_packed, proj.scales, groupsize, out=buf[1:m + 1]).clone()

    outs = [run(), run()]
    lib.kiln_w4a16_set_small_batch_kernel(0)
    try:
        decode = run()
    finally:
        lib.kiln_w4a16_set_small_batch_kernel(1)
    torch.cuda.synchronize()
    assert lib.kiln_w4a16_check_device_status(None, None) == 0
    assert (buf[0] == 3.0).all() and (buf[m + 1] == 3.0).all()
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    assert rel_err(from_torch_bf16(outs[0]), ref.astype(np.float32)) <= REL_TOL
    norm = lambda t: float(np.linalg.norm(from_torch_bf16(t).astype(np.float64) - ref))
    assert norm(outs[0]) <= 1.02 * norm(decode), "less precise than the decode kernel"


@pytest.mark.parametrize("m,k,n_half", [(9, 2560, 9216), (16, 128, 256), (200, 640, 512)])
def test_swiglu_in_its_epilogue(cuda_device, m, k, n_half):
    a, fused, g, u = _gate_up_case(m, k, n_half, seed=m, dev=cuda_device)
    out = kiln_b200.swiglu_gate_up(to_torch_bf16(a, cuda_device), fused)
    torch.cuda.synchronize()
    assert rel_err(from_torch_bf16(out), (_silu(g) * u).astype(np.float32)) <= REL_TOL
