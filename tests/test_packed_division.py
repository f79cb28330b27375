"""The divisions by 7 and 127 of the momentum codecs (csrc/kaon_packed.cuh: quotient by the rounded reciprocal, exact
residual, one correction), restated in long double: the correctly rounded quotient for every mantissa.  Scaling the
dividend by a power of two scales every step exactly, within 1e-12 <= a < 2^128 no step is subnormal and none overflows, so
one binade of dividends stands for all."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-optimizers_b200", "csrc")


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs an extended long double")
@pytest.mark.parametrize("d", [7, 127])
def test_division_by_a_constant_is_correctly_rounded(d):
    text = open(os.path.join(CSRC, "kaon_packed.cuh")).read()
    lit = re.search(r"const float r%d = ([0-9.]+)f;" % d, text).group(1)
    r = np.float32(lit)
    assert r == np.float32(1.0) / np.float32(d)
    f = re.search(r"float div%d_exact\(float a\) \{(.*?)\n\}" % d, text, flags=re.S).group(1)
    assert "__fmul_rn(a, r%d)" % d in f and "__fmaf_rn(__fmaf_rn(-%d.0f, q0, a), r%d, q0)" % (d, d) in f
    for top in range(0, 1 << 23, 1 << 20):   # a in [1, 2), a chunk at a time
        bits = np.arange(top, top + (1 << 20), dtype=np.uint32) | np.uint32(0x3F800000)
        a = bits.view(np.float32)
        q0 = a * r                                                    # one rounding, to fp32
        wide = np.longdouble
        res = (wide(-d) * q0.astype(wide) + a.astype(wide))          # exact: 24 + 7 bits
        assert np.array_equal(res.astype(np.float32).astype(wide), res)   # and an fp32 number, as the FMA leaves it
        q = (res * wide(r) + q0.astype(wide)).astype(np.float32)     # the last FMA: a sum of at most 64 bits, rounded once
        assert np.array_equal(q, a / np.float32(d)), top
