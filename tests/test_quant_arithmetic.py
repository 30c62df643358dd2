"""Arithmetic of the quantiser's kernels that replaces a division, checked for every significand on the host."""
import numpy as np


def test_row_scale_quotient_for_every_significand():
    """a / 127 from RN(1 / 127): q = RN(a y), then one Markstein step RN(q + RN(a - 127 q) y), as csrc/quant_common.cuh
    computes the row scale. Both fused operations are formed exactly (products in float64, the last sum as two
    float64 parts) and rounded once; the result has to be the IEEE quotient for all 2^23 significands. A binade
    stands for all: nothing here leaves the normal range while a is above 2^-90."""
    y = np.float32(1.0) / np.float32(127.0)
    a = (np.arange(1 << 23, dtype=np.uint32) + np.uint32(0x3F800000)).view(np.float32)
    q = a * y
    residual = (a.astype(np.float64) - 127.0 * q.astype(np.float64)).astype(np.float32)  # exact before the rounding
    # q + residual * y in one rounding: the product has 48 bits, so it is exact; the sum is rounded to float64 with its
    # error term (two-sum), and the float32 rounding may only be decided where that error cannot cross a boundary
    product = residual.astype(np.float64) * np.float64(y)
    big = q.astype(np.float64)
    total = big + product
    error = (big - (total - (total - big))) + (product - (total - big))
    rounded = total.astype(np.float32)
    halfway = np.abs(total - rounded.astype(np.float64)) * 2 == np.spacing(rounded).astype(np.float64)
    assert not np.any(halfway & (error != 0))
    want = (a.astype(np.float64) / 127.0).astype(np.float32)  # no quotient by 127 is within 2^-33 of a boundary
    assert np.array_equal(rounded, want)


def test_bf16_quotient_for_every_pair_of_significands():
    """bf16(v / s) from RN(v RN(1 / s)) for all 128 x 128 pairs of 8-bit significands (div2_bf16)."""
    v = np.arange(128, 256, dtype=np.float32)[:, None]
    s = np.arange(128, 256, dtype=np.float32)[None, :]

    def bf16(x):
        bits = x.astype(np.float32).view(np.uint32)
        return (bits + np.uint32(0x7FFF) + ((bits >> np.uint32(16)) & np.uint32(1))) >> np.uint32(16)

    product = v * (np.float32(1.0) / s)
    assert np.array_equal(bf16(product), bf16((v.astype(np.float64) / s.astype(np.float64)).astype(np.float32)))
