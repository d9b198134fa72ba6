"""The vectorised host packer where it could differ from the scalar one: ties between quantisation steps and their neighbours,
NaN, infinities, zero and subnormal scales, group sizes that are not 128, the smallest matrix and one with several column
blocks.  Bit-exact with the oracle."""
import numpy as np
import pytest

import kiln_b200
from oracle import C
from tests.test_gpu_pack_edges import _edge_weight


@pytest.mark.parametrize("k,n,gs", [(128, 256, 128), (640, 768, 128), (256, 512, -1), (256, 256, 32), (384, 256, 384)])
@pytest.mark.parametrize("threads", [1, 3])
def test_host_pack_at_ties_and_special_values(k, n, gs, threads):
    w = _edge_weight(k, n, False).numpy()
    p, s, d = kiln_b200.pack.quantize_and_pack(w, k, n, gs, num_threads=threads)
    po, so, do, _ = C.quantize_and_pack(w, gs)
    assert (s.view(np.uint16) == so.view(np.uint16)).all()
    assert (p == po).all()
    assert np.array_equal(d.view(np.uint32)[~np.isnan(do)], do.view(np.uint32)[~np.isnan(do)])
