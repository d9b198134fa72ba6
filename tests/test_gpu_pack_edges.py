"""Device packer where its arithmetic could go wrong: quotients on and next to the ties between two quantisation steps,
NaN, infinities, zero and subnormal scales, and both group sizes in both weight types.  Bit-exact with the host packer, which
divides and rounds every weight."""
import numpy as np
import pytest
import torch

import kiln_b200
from tests.test_gpu_packer import _dev_pack

pytestmark = pytest.mark.gpu


def _edge_weight(k, n, bf16):
    rng = np.random.default_rng(k + n)
    w = (rng.standard_normal((k, n)) * 0.02).astype(np.float32)
    # columns whose maximum makes the scale exactly 2^-6: quotients in steps of a quarter hit every tie, next to it the
    # neighbouring floats on both sides
    steps = rng.integers(-30, 31, (k, 64)).astype(np.float32) / 4
    w[:, :64] = np.clip(steps, -7.5, 7.5) * np.float32(2.0 ** -6)
    w[::128, :64] = np.float32(7.5 * 2.0 ** -6)
    w[1::4, :64] = np.nextafter(w[1::4, :64], np.float32(np.inf))
    w[2::4, :64] = np.nextafter(w[2::4, :64], np.float32(-np.inf))
    w[::128, :64] = np.float32(7.5 * 2.0 ** -6)
    w[3, 70] = np.nan
    w[5, 71] = np.inf
    w[6, 72] = -np.inf
    w[:, 73] = 0
    w[:, 74] *= 1e-6  # subnormal scale
    w[:, 75] *= 1e-9  # scale rounds to zero
    w[:, 76] *= 1e8   # scale overflows
    w[7, 77] = np.float32(3e38)
    w[:, 78] = -np.abs(w[:, 78])
    t = torch.from_numpy(w)
    return t.to(torch.bfloat16) if bf16 else t


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("k,n,gs", [(128, 256, 128), (640, 768, 128), (128, 256, -1), (1152, 512, -1)])
def test_device_pack_at_ties_and_special_values(cuda_device, k, n, gs, bf16):
    w = _edge_weight(k, n, bf16)
    p, s, d = _dev_pack(w.to(cuda_device), gs)
    p2, s2, d2 = kiln_b200.pack.quantize_and_pack(w.float().numpy(), k, n, gs)
    assert (s == s2.view(np.uint16)).all()
    assert (p == p2).all()
    assert np.array_equal(d, d2, equal_nan=True)


@pytest.mark.parametrize("k,n,gs", [(128, 256, 128), (640, 512, -1), (4224, 256, 128)])
def test_gptq_repack_sizes(cuda_device, k, n, gs):
    """One 16-row tile group, a partial last block of tiles, more tiles than a block takes."""
    import oracle

    rng = np.random.default_rng(k)
    q = rng.integers(0, 16, (k, n), dtype=np.uint8)
    rows = 1 if gs == -1 else k // gs
    s = (0.01 * np.abs(rng.standard_normal((rows, n))) + 1e-3).astype(np.float16)
    qw, qz = oracle.np_gptq_pack(q, np.full((rows, n), 8, np.uint8))
    t = lambda a: torch.from_numpy(a).to(cuda_device)
    proj = kiln_b200.pack_from_gptq(t(qw), t(qz), t(s), gs)
    assert (proj.b_packed.cpu().numpy() == oracle.C.pack_nibbles(q)).all()
    assert (proj.scales.cpu().view(torch.int16).numpy().view(np.uint16) == oracle.C.permute_scales(s, gs).view(np.uint16)).all()
