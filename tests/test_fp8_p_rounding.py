"""f16(e4m3(448 p) / 448) as the kernels compute it, in f16 arithmetic: the quotient by the rounded reciprocal, its exact
remainder, one correction.  Enumerated over all codes, against the correctly rounded quotient."""
import numpy as np
import torch


def test_division_by_448_in_half_precision_is_correctly_rounded():
    codes = torch.arange(0, 127, dtype=torch.uint8).view(torch.float8_e4m3fn).double().numpy()
    half = lambda x: x.astype(np.float16).astype(np.float64)         # a fused operation: exact in fp64, rounded once
    inv = np.float64(np.uint16(0x1892).view(np.float16))
    assert inv == np.float64(np.float16(1 / 448))
    q = half(codes * inv)
    q = half(q + half(codes - 448 * q) * inv)
    assert (q == half(codes / 448)).all()
