"""How the tcgen05 kernels turn packed nibbles into bf16 weights, restated with numpy (no GPU): a nibble, read as a bf16 where it sits, times
s * 2^133 or s * 2^129, less 8 s, in one fused multiply-add, everything at 2^-22 of its value (kiln_b200/csrc/w4a16_common.cuh)."""
import re
from pathlib import Path

import numpy as np

_SRC = (Path(__file__).parent.parent / "kiln_b200" / "csrc" / "w4a16_common.cuh").read_text()


def _constant(name):
    """A number as the source has it: 0x77007700u, 4194304.f, 1.f / 4194304.f."""
    text = re.search(r"\b" + name + r" = ([^,;]+)[,;]", _SRC).group(1)
    value = 1.0
    for i, part in enumerate(text.split("/")):
        number = float(int(part.strip().rstrip("u"), 16)) if "0x" in part else float(part.strip().rstrip("f"))
        value = number if i == 0 else value / number
    return value


def _bf16_pair(name):
    """The value of a bf16x2 constant, whose halves must be alike."""
    bits = int(_constant(name))
    assert bits >> 16 == bits & 0xFFFF
    return float(np.array([bits & 0xFFFF0000], dtype=np.uint32).view(np.float32)[0])


def test_the_constants_of_the_source():
    assert int(_constant("kNibMask")) == 0x000F000F and int(_constant("kHiNibMask")) == 0x00F000F0
    factor = _constant("kWeightFactor")
    assert factor == 2.0 ** -22 and _constant("kWeightUnscale") == 2.0 ** 22
    assert _bf16_pair("lo") * 2.0 ** -133 == factor and _bf16_pair("hi") * 2.0 ** -129 == factor and _bf16_pair("off") == -8.0 * factor


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
    lo, hi, off = s * _bf16_pair("lo"), s * _bf16_pair("hi"), s * _bf16_pair("off")
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
