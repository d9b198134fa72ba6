"""SwiGLU where its parts are easy to lose: per-column scales (group size -1), whose gate and up columns meet in an epilogue with scales of
their own (against the fp64 oracle, max|out - ref| / max|ref| <= 1e-2), and gates near the end of the exponential's range."""
import numpy as np
import pytest
import torch

import kiln_b200
import oracle
from kiln_b200 import _lib
from oracle import C
from tests.test_gpu_epilogue import _proj, _silu
from tests.util import REL_TOL, from_torch_bf16, rel_err, to_torch_bf16

pytestmark = pytest.mark.gpu


# decode kernel; the small-batch kernel's fp32-scale variant from its smallest problem to its most rows, K of one stage and of more
# than the teams; the small-batch kernel itself, 64 and 128 rows; CTA pairs
@pytest.mark.parametrize("m,k,n_half", [(1, 2560, 512), (5, 640, 512), (9, 128, 128), (13, 2560, 256), (16, 9216, 1280), (17, 640, 384),
                                        (129, 1536, 384), (256, 640, 512), (24, 2560, 9216), (64, 2560, 9216), (100, 640, 9216), (300, 1152, 512)])
def test_each_column_keeps_its_own_scale(cuda_device, m, k, n_half):
    a, qg, sg = oracle.synth_inputs(m, k, n_half, seed=m + k, groupsize=-1)
    _, qu, su = oracle.synth_inputs(1, k, n_half, seed=m + k + 1, groupsize=-1)
    fused = kiln_b200.interleave_gate_up(_proj(qg, sg, -1, cuda_device), _proj(qu, su, -1, cuda_device))
    out = kiln_b200.swiglu_gate_up(to_torch_bf16(a, cuda_device), fused)
    torch.cuda.synchronize()
    assert _lib.lib().kiln_w4a16_check_device_status(None, None) == 0
    ref = _silu(C.gemm_fp64(a, qg, sg, -1).astype(np.float64)) * C.gemm_fp64(a, qu, su, -1).astype(np.float64)
    assert rel_err(from_torch_bf16(out), ref.astype(np.float32)) <= REL_TOL


@pytest.mark.parametrize("m", [8, 9, 16])
def test_silu_of_a_gate_near_its_underflow(cuda_device, m):
    """gate = -87.5 .. -88.5: 1 + exp(-gate) lies above 2^126, where an approximate quotient is 0 and silu(gate) * up is still a normal
    number of about 1e-35.  Relative error: half a unit of bf16, whose
    eight-bit significand makes that at most 2^-8, plus the exponential's 2 + 1.173 * 88 units of fp32 (1e-5)."""
    k, n_half = 128, 128
    qg, qu = np.zeros((k, n_half), np.uint8), np.zeros((k, n_half), np.uint8)
    qg[:], qu[:] = 8, 8          # zero, but for the first row: gate 7 x, up x
    qg[0], qu[0] = 15, 9
    s = np.ones((1, n_half), np.float16)
    x = np.zeros((m, k), np.float32)
    x[:, 0] = np.linspace(-12.64, -12.5, m)
    x_t = torch.from_numpy(x).to(torch.bfloat16)
    fused = kiln_b200.interleave_gate_up(_proj(qg, s, 128, cuda_device), _proj(qu, s, 128, cuda_device))
    out = from_torch_bf16(kiln_b200.swiglu_gate_up(x_t.to(cuda_device), fused)).astype(np.float64)
    v = x_t[:, 0].double().numpy()
    ref = (7 * v / (1 + np.exp(-7 * v)) * v)[:, None]
    assert np.abs(out / ref - 1).max() <= 2.0 ** -8 + 2e-5


# the kernel of CTA pairs, 256 and 128 columns a tile
@pytest.mark.parametrize("groupsize", [128, -1])
@pytest.mark.parametrize("m,n_half", [(129, 1024), (300, 1024), (512, 9216)])
def test_extreme_gates_and_ups_of_the_pair_kernel(cuda_device, m, n_half, groupsize):
    """No step from the sums to silu(gate) * up may overflow or vanish where the result does not.  Relative error: half a unit of bf16 (at most
    2^-8), the exponential's error for |gate| up to 88 (2e-5, as above), and 2^-128, half of fp32's last bit at the weights' factor of 2^-22.  Zeros
    and infinities are exact."""
    k = 256
    q = np.full((k, n_half), 8, np.uint8)
    qg, qu = q.copy(), q.copy()
    qg[0], qu[1] = 9, 9          # gate = x[0], up = x[1]
    s = np.ones((1 if groupsize == -1 else 2, n_half), np.float16)
    pairs = [(1e32, 1.0), (1e32, 0.0), (1e35, -1e-10), (3e38, 1e-30), (3e38, 1.0), (1e30, 1e30), (-87.0, 1.0), (-87.0, 40.0), (-60.0, 1e-6), (-20.0, 1e30),
             (-1e5, 1e5), (0.0, 7.0), (1e-30, 1.0), (50.0, 1e-30), (2.0, 3e38), (-0.5, 0.25), (5.0, -3.0)]
    x = torch.zeros((m, k))
    x[:, :2] = torch.tensor([pairs[i % len(pairs)] for i in range(m)])
    x = x.bfloat16()
    fused = kiln_b200.interleave_gate_up(_proj(qg, s, groupsize, cuda_device), _proj(qu, s, groupsize, cuda_device))
    out = kiln_b200.swiglu_gate_up(x.to(cuda_device), fused).cpu().double().numpy()
    assert _lib.lib().kiln_w4a16_check_device_status(None, None) == 0
    g, u = x[:, 0].double().numpy(), x[:, 1].double().numpy()
    with np.errstate(over="ignore"):
        ref = (g / (1.0 + np.exp(-g)) * u)[:, None] * np.ones((1, n_half))
    large = np.abs(ref) > 3.4e38
    exact = large | (np.abs(ref) < 2.0 ** -149)
    want = np.where(exact, 0.0, ref)
    want[large] = np.sign(ref[large]) * np.inf
    assert (out[exact] == want[exact]).all()
    assert (np.abs(out[~exact] - want[~exact]) <= np.abs(want[~exact]) * (2.0 ** -8 + 2e-5) + 2.0 ** -128).all()
