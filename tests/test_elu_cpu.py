"""The ELU of the codec's epilogues is written from exp's Taylor series near zero and from CUDA's expf below -1/2.  Its coefficients are
read from the source and the series evaluated in fp32 against expm1 in 64 bits."""
import math
import os
import re

import numpy as np

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vui_b200", "csrc")


def test_elu_series_and_its_error():
    src = open(os.path.join(CSRC, "split_gemm.cuh")).read()
    body = src[src.index("if (act == SA_ELU)"):src.index("if (act == SA_GELU)")]
    coef = [float(np.float32(1) / np.float32(d)) for d in re.findall(r"1\.f / (\d+)\.f", body)] + [0.5]
    assert "p = fmaf(p, v, 0.5f)" in body and "near = fmaf(v * v, p, v), far = expf(v) - 1.f" in body and "v > -0.5f ? near : far" in body
    assert coef == [float(np.float32(1.0 / math.factorial(n))) for n in range(9, 1, -1)]
    fma = lambda a, b, c: (a.astype(np.float64) * b + c).astype(np.float32)  # noqa: E731  one rounding
    v = -np.exp(np.linspace(math.log(1e-30), math.log(0.5), 200001)).astype(np.float32)
    p = np.full_like(v, coef[0])
    for c in coef[1:]:
        p = fma(p, v, np.float32(c))
    near = fma(v * v, p, v)
    want = np.expm1(v.astype(np.float64))
    # the terms left out are below v^9 / 10! = 6e-10 of v; the square, the sum and p, whose share is at most a quarter, round to 6e-8 each
    assert (np.abs(near - want) / np.abs(want)).max() < 1.5e-7
    # below -1/2 one rounding of expf (2 ulp of at most 0.61) and one of the difference, of a value of at least 0.39
    far = (np.exp(np.linspace(-100, -0.5, 200001)).astype(np.float32) - np.float32(1)).astype(np.float64)
    assert np.abs(far - np.expm1(np.linspace(-100, -0.5, 200001))).max() < 1.2e-7
