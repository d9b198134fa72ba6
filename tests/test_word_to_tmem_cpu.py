"""From a packed word to tensor memory in the small-batch tcgen05 kernel (kiln_b200/csrc/smallm_w4a16_tmem.cu), restated with numpy and checked
against the oracle's packer on the CPU.

Lane (c, qd) of a warp holds two words per 16-row K tile.  Four shifts and masks give a word's four registers, and tcgen05.st.16x128b puts
register 0 of lane (c, qd) into TMEM lane c, cell qd, register 1 into lane c + 8, the next two into cells 4 + qd of the same lanes; the
first word goes to TMEM lanes 0..15 of the warp's quarter, the second to lanes 16..31.  A cell is a K pair of the lane's weight column.
Plain: words 2h and 2h + 1, lane = column 32h + lane; with SwiGLU words h and h + 2, so that a gate column of a chunk (gate and up alternate in
runs of 32) and its up column are sixteen lanes apart."""
import numpy as np
import pytest

from oracle import C


def _column(swiglu, h):
    lane = np.arange(32)
    return 16 * h + lane % 16 + 32 * (lane // 16) if swiglu else 32 * h + lane


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("h", [0, 1])
def test_each_tmem_lane_gets_one_column(h, swiglu):
    q = np.random.default_rng(7 + h).integers(0, 16, size=(16, 64), dtype=np.uint8)  # one K tile x one 64-column chunk of nibbles
    block = np.asarray(C.pack_nibbles(q)).view(np.uint32).reshape(32, 4)                # 512 bytes: lane L holds words 4L .. 4L+3
    lane = np.arange(32)
    c, qd = lane >> 2, lane & 3
    tmem = np.full((32, 8, 2), 255, dtype=np.uint8)                                     # [TMEM lane][cell][half of the pair]
    for half, word in enumerate((h, h + 2) if swiglu else (2 * h, 2 * h + 1)):
        x = block[:, word]
        for reg, shift in enumerate((0, 8, 4, 12)):
            v = (x >> np.uint32(shift)) & np.uint32(0x000F000F)
            row, cell = 16 * half + c + 8 * (reg & 1), qd + 4 * (reg >> 1)
            tmem[row, cell, 0], tmem[row, cell, 1] = v & 0xF, v >> 16
    want = q[:, _column(swiglu, h)].T.reshape(32, 8, 2)                                 # K pair `cell` of the lane's column
    assert np.array_equal(tmem, want)


def test_swiglu_partners_are_sixteen_lanes_apart():
    for h in (0, 1):
        col = _column(True, h)
        assert (col[:16] < 32).all() and (col[16:] == col[:16] + 32).all()
    for swiglu in (False, True):  # the two warps of a chunk cover its columns once
        assert sorted(np.concatenate([_column(swiglu, 0), _column(swiglu, 1)])) == list(range(64))


def test_scales_of_a_lane():
    """Position 8i + j of a chunk's scale order holds column 8j + i (kiln-marlin-gemm/src/lib.rs:333-341): the scales of a word's columns c and
    c + 8 are neighbours, at 8c + 2 * word; and that of the column that a TMEM lane finishes is at 8 * (column % 8) + column / 8."""
    s = np.arange(64, dtype=np.float32).reshape(1, 64) + 1.0  # scale value = natural column + 1
    perm = np.asarray(C.permute_scales(s.astype(np.float16), 128)).astype(np.float32).reshape(64)
    for swiglu in (False, True):
        for h in (0, 1):
            for c in range(8):
                for i in range(2):
                    at = 8 * c + (2 if swiglu else 4) * h + (4 if swiglu else 2) * i
                    word = h + 2 * i if swiglu else 2 * h + i
                    assert perm[at] == 16 * word + c + 1 and perm[at + 1] == 16 * word + c + 8 + 1
            for col in _column(swiglu, h):
                assert perm[8 * (col & 7) + (col >> 3)] == col + 1
