"""GPTQ repack on the device: zero-points that are not 8 are counted wherever they sit, and the scales of every row reach their places, for
numbers of scale rows below, at and above what the blocks of a column take at a time."""
import numpy as np
import pytest
import torch

from kiln_b200 import _lib
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n,g", [(128, 64, 128), (512, 256, -1), (1024, 128, 16), (640, 320, 32), (4224, 256, 128), (16, 64, 16)])
def test_counts_and_scales(cuda_device, k, n, g):
    rng = np.random.default_rng(k + n)
    rows = 1 if g == -1 else k // g
    q = rng.integers(0, 16, (k, n), dtype=np.uint8)
    s = rng.integers(0, 1 << 16, (rows, n), dtype=np.uint16)
    lib = _lib.lib()
    for bad in ([], [(0, 0)], [(rows - 1, n - 1)], [(rows // 2, n // 2), (rows - 1, 0), (0, n - 1)]):
        zeros = np.full((rows, n), 8, np.uint8)
        for r, c in bad:
            zeros[r, c] = rng.integers(0, 8)
        qw, qz = oracle.np_gptq_pack(q, zeros)
        t = lambda a: torch.from_numpy(a).to(cuda_device)
        qw_t, qz_t, s_t = t(qw), t(qz), t(s.view(np.int16))
        b = torch.empty(k // 16 * 2 * n, dtype=torch.int32, device=cuda_device)
        out = torch.empty(rows * n, dtype=torch.int16, device=cuda_device)
        count = torch.full((1,), 77, dtype=torch.int32, device=cuda_device)
        args = (qw_t.data_ptr(), qz_t.data_ptr(), s_t.data_ptr(), k, n, g, b.data_ptr(), out.data_ptr())
        assert lib.kiln_w4a16_repack_gptq_device(*args, count.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert int(count) == len(set(bad))
        want = oracle.C.permute_scales(s.view(np.float16), g if g == -1 else 128).view(np.uint16).reshape(-1)
        assert (out.cpu().numpy().view(np.uint16) == want).all()
        assert (b.cpu().numpy() == oracle.C.pack_nibbles(q).reshape(-1)).all()
        assert lib.kiln_w4a16_repack_gptq_device(*args, None, None) == 0  # (nobody asks for the count)
        torch.cuda.synchronize()
