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


def test_bf16_quotient_in_two_bf16_parts_for_every_pair_of_significands():
    """bf16(v / s) as fma(v, r1, bf16(v r2)) rounded once to bf16, with r1 = bf16(r), r2 = bf16(r - r1), as SplitReciprocal of
    csrc/quant_common.cuh forms it, for all 128 x 128 pairs and every fp32 r between 1 + 2^-25 and 1 + 43 / 2^25 times the
    exact reciprocal. The kernel's r is 1 + 6 / 2^23 times an approximate one within 2^-23 of the exact one, rounded once
    more: between 1 + 18 / 2^25 and 1 + 30 / 2^25 times."""
    def bf16(x):  # nearest even, 8 significant bits; x exact in float64
        m, e = np.frexp(x)
        return np.ldexp(np.rint(m * 256.0), e - 8)

    v = np.arange(128, 256, dtype=np.float64)
    seen = 0
    for s in range(128, 256):
        want = bf16(v / s)  # no quotient is within 2^-17 of a rounding boundary
        least, most = ((1.0 + step * 2.0 ** -25) / s for step in (1, 43))
        bits = np.float32([least, most]).view(np.uint32)
        r = np.arange(bits[0] - 1, bits[1] + 2, dtype=np.uint32).view(np.float32).astype(np.float64)
        r = r[(r >= least) & (r <= most)]
        seen += len(r)
        r1 = bf16(r)
        r2 = bf16(r - r1)  # the difference is exact
        got = bf16(v[:, None] * r1 + bf16(v[:, None] * r2))  # 8 + 8 bits and a term at most 2^9 times smaller: exact in float64
        assert np.array_equal(got, np.broadcast_to(want[:, None], got.shape)), s
    assert seen >= 128 * 10  # an fp32 step is 2^-24 to 2^-23 of the reciprocal


def test_direct_codes_from_one_product_for_every_pair_of_significands():
    """direct_codes of csrc/quant_common.cuh: the nearest even integer to v y against that to the IEEE quotient
    RN(v / scale), scale = RN(maximum / 127), for every significand of the maximum, every significand of v (fewer bits
    too) and every exponent that gives a code, with y up to 2^-22 of itself away from the one computed (the approximate
    reciprocal, its Newton step and the roundings of the move leave less) unless the scale is a power of two."""
    f32 = np.float32
    for M in range(128, 256):
        scale = f32(np.float64(M) / 127.0)  # no quotient by 127 is near a boundary of fp32
        apart = 127.0 * np.float64(scale) - M  # exact
        assert (apart == 0.0) == (M == 254)
        move = 0.0 if apart == 0.0 else 2.0 ** -21 if apart <= M * 3.0e-8 else -2.0 ** -21
        y = np.float64(f32(1.0 / np.float64(scale))) * (1.0 + move)
        for k in range(10):  # beyond, v is below a quarter of the scale
            v = np.arange(1, 256, dtype=np.float64) * 2.0 ** -k
            v = v[v <= M]
            want = np.rint((v / np.float64(scale)).astype(f32))
            for wobble in (0.0,) if M == 254 else (-2.0 ** -22, 0.0, 2.0 ** -22):
                got = np.rint((v * np.float64(f32(y * (1.0 + wobble)))).astype(f32))
                assert np.array_equal(want, got), (M, k, wobble)
