"""GPTQ repack through the C ABI into int32 buffers that are aligned to a word and no more (a slice of an arena, say): the same words as into an
aligned one, and none outside the buffer."""
import numpy as np
import pytest
import torch

import oracle
from kiln_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("k,n", [(128, 256), (640, 320)])
def test_gptq_repack_into_a_word_aligned_buffer(cuda_device, k, n, offset):
    rng = np.random.default_rng(k + offset)
    q = rng.integers(0, 16, (k, n), dtype=np.uint8)
    s = (0.01 * np.abs(rng.standard_normal((k // 128, n))) + 1e-3).astype(np.float16)
    qw, qz = oracle.np_gptq_pack(q, np.full((k // 128, n), 8, np.uint8))
    t = lambda a: torch.from_numpy(a).to(cuda_device)
    qw_t, qz_t, s_t = t(qw), t(qz), t(s)
    words = k // 16 * 2 * n
    buf = torch.full((words + 8,), 0x5A5A5A5A, dtype=torch.int32, device=cuda_device)
    sp, bad = torch.empty_like(s_t), torch.empty(1, dtype=torch.int32, device=cuda_device)
    assert buf.data_ptr() % 16 == 0
    rc = _lib.lib().kiln_w4a16_repack_gptq_device(qw_t.data_ptr(), qz_t.data_ptr(), s_t.data_ptr(), k, n, 128, buf.data_ptr() + 4 * offset, sp.data_ptr(),
                                                  bad.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and bad.item() == 0
    got = buf.cpu().numpy()
    assert (got[offset:offset + words].reshape(k // 16, 2 * n) == oracle.C.pack_nibbles(q)).all()
    assert (got[:offset] == 0x5A5A5A5A).all() and (got[offset + words:] == 0x5A5A5A5A).all()
