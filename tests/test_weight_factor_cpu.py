"""How the tcgen05 kernels turn packed nibbles into bf16 weights, restated with numpy (no GPU): a nibble, read as a bf16 where it sits, times
s * 2^133 or s * 2^129, less 8 s, in one fused multiply-add, everything at 2^-22 of its value (kiln_b200/csrc/w4a16_common.cuh)."""
import numpy as np


def _bf16_bits(x):
    """float64 -> bf16 bits, one rounding to nearest even (for values that are normal bf16 numbers, or zero)."""
    m, e = np.frexp(np.asarray(x, dtype=np.float64))
    q = np.rint(m * 256.0)  # 8 significant bits, ties to even
    return q * np.exp2(e.astype(np.float64) - 8.0)


def test_a_nibble_where_it_sits_is_a_linear_scale_of_bf16():
    nib = np.arange(16, dtype=np.uint32)
    lo = (nib << 16).view(np.float32).astype(np.float64)          # bits 0..3 of a half: subnormals
    hi = ((nib << 4) << 16).view(np.float32).astype(np.float64)   # bits 4..7: into the first binade of the normals
    assert np.array_equal(lo, nib * 2.0 ** -133)
    assert np.array_equal(hi, nib * 2.0 ** -129)


def test_fused_multiply_add_rounds_as_subtract_and_multiply_do_for_every_fp16_scale():
    h = np.arange(0, 0x7C00, dtype=np.uint16).view(np.float16)    # zero, subnormals, normals; signs are symmetric
    s = _bf16_bits(h.astype(np.float64))
    lo, hi, off = s * 2.0 ** 111, s * 2.0 ** 107, -8.0 * s * 2.0 ** -22
    largest = (2.0 - 2.0 ** -7) * 2.0 ** 127
    assert lo.max() <= largest and hi.max() <= largest
    smallest = 2.0 ** -126
    assert hi[1:].min() >= smallest and np.abs(off[1:]).min() >= smallest
    for n in range(16):
        want = _bf16_bits((n - 8.0) * s) * 2.0 ** -22             # (n - 8 and the product of eight-bit numbers are exact in float64)
        for bits, mul in ((n, lo), (n << 4, hi)):
            x = float((np.array([bits], dtype=np.uint32) << 16).view(np.float32)[0])
            got = _bf16_bits(x * mul + off)                       # exact in float64: at most 12 + 8 bits
            assert np.array_equal(got, want)
        assert n == 8 or np.abs(want[1:]).min() >= smallest
