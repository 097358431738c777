"""The integer arithmetic of the decode kernel, restated in numpy (no GPU).

A unit is one token's 256 products p = s_in * x of a chunk.  With m = max |p| and the class j = (column % 256) / 32, a
column becomes Z = round(p * 32500 / m * 2^(7-j)), negated for j = 7, by adding 1.5 * 2^23 in fp32; the low mantissa bits
of that sum, 0x8080 added, are the three signed bytes of Z.  The kernel feeds `word & (0x01010101 << j)` (an int8x4 with
values {0, 2^j}, {0, -128} for j = 7) to an s8 MMA against the bytes, so every class has the weight 128 * p * 32500 / m,
and sum(+-p) = unit * (sum - 2 * S) with unit = m / (128 * 32500), S the sum over the set bits, both modulo 2^32.
"""
import numpy as np

Q_MAX = 32500
MAGIC = np.float32(12582912.0 + 32896.0)      # 1.5 * 2^23 + 0x8080
J = np.arange(256) // 32
A = np.where(J == 7, -128, 1 << J)            # what a set bit of class j is worth to the MMA


def words_of(p):
    """fp32 words of the conversion, and m, for the 256 products of a unit (finite, m above 1e-31)."""
    m = np.float32(np.abs(p).max())
    inv = np.float32(Q_MAX) * (np.float32(1) / m)
    inv_j = inv * np.where(J == 7, np.float32(-1), np.float32(2.0) ** (7 - J)).astype(np.float32)
    # the product of two fp32 numbers is exact in fp64; the sum is rounded to an integer by the size of MAGIC
    y = (p.astype(np.float64) * inv_j.astype(np.float64) + np.float64(MAGIC)).astype(np.float32)
    return y.view(np.uint32), m


def bytes_of(w):
    """The kernel's three bytes of a word, as signed values: packed adds and exclusive ors, without carries between bytes."""
    s8 = lambda b: ((b & 0xFF).astype(np.int64) ^ 0x80) - 0x80
    b2 = (w >> 16) & 0xFF
    assert np.all(b2 + 0x40 <= 0xFF)           # the packed addition of 0x40404040 carries nothing into a neighbour
    return s8((w & 0xFF) ^ 0x80), s8(((w >> 8) & 0xFF) ^ 0x80), s8((b2 + 0x40) ^ 0x80)


def test_three_signed_bytes_recombine_for_every_integer():
    most = int(Q_MAX * 128 * (1 + 2.0 ** -20)) + 1       # the reciprocal and its products are rounded
    assert most < 2 ** 22
    z = np.arange(-most, most + 1, dtype=np.int64)
    w = (np.float32(12582912.0) + (z + 0x8080).astype(np.float32)).view(np.uint32)
    assert np.array_equal(w, (0x4B400000 + 0x8080 + z).astype(np.uint32))
    b0, b1, b2 = bytes_of(w)
    assert np.array_equal(65536 * b2 + 256 * b1 + b0, z)


def unit_of(p):
    """{unit value, sum} and the three byte rows, as quantise_unit leaves them in shared memory."""
    w, m = words_of(p)
    lanes = w.reshape(32, 8).astype(np.uint64).sum(axis=1)
    part = (lanes - 8 * (0x4B400000 + 0x8080)).astype(np.uint32).view(np.int32).astype(np.int64)      # modulo 2^32, per lane
    part = part * A[::8]
    assert np.abs(part).max() <= 2 ** 25
    total = int(part.sum())
    assert abs(total) < 2 ** 30
    return np.float32(m) * np.float32(1.0 / (128 * Q_MAX)), total, bytes_of(w)


def products(seed, n=256):
    g = np.random.default_rng(seed)
    p = (g.standard_normal(n) * 10.0 ** g.uniform(-8, 8)).astype(np.float32)
    p[g.integers(n, size=seed % 64)] = 0
    return p


def test_sums_over_signs_are_exact_and_in_range():
    for seed in range(40):
        p = products(seed) if seed else np.full(256, 3.0, np.float32)      # seed 0: every column at the bound
        unit, total, (b0, b1, b2) = unit_of(p)
        z = 65536 * b2 + 256 * b1 + b0
        assert np.abs(A * z).sum() < 2 ** 30
        bits = np.random.default_rng(seed).integers(0, 2, size=(64, 256)).astype(np.int64)
        bits[0], bits[1] = 0, 1
        c0, c1, c2 = (bits * A) @ b0, (bits * A) @ b1, (bits * A) @ b2
        assert max(np.abs(c).max() for c in (c0, c1, c2)) < 2 ** 31         # int32 accumulators
        S = (c0 + (c1 << 8) + (c2 << 16)) & 0xFFFFFFFF
        got = ((total - 2 * S) & 0xFFFFFFFF).astype(np.uint32).view(np.int32).astype(np.int64)
        assert np.array_equal(got, ((1 - 2 * bits) * (A * z)).sum(axis=1))


def test_quantisation_error():
    for seed in range(1, 40):
        p = products(seed)
        unit, _, (b0, b1, b2) = unit_of(p)
        q = (A * (65536 * b2 + 256 * b1 + b0)) * np.float64(unit)
        # half an integer of class j is 2^j / 2 <= 64 of 128 * 32500 units; the rest is the rounding of reciprocal and unit
        assert np.abs(q - p).max() <= np.abs(p).max() * (64 / (128 * Q_MAX) + 2.0 ** -21)


def test_small_products_scaled_by_a_power_of_two_give_the_same_integers():
    # below 1e-31 the reciprocal of the maximum times 32500 * 128 would overflow fp32
    assert np.float32(Q_MAX) * (np.float32(1) / np.float32(1e-31)) * np.float32(128) < np.finfo(np.float32).max
    p = (products(3) / np.abs(products(3)).max()).astype(np.float32)
    tiny = p * np.float32(2.0 ** -110)
    assert np.abs(tiny).max() <= 1e-31
    want, _ = words_of(p)
    got, m = words_of(tiny * np.float32(2.0 ** 64))
    assert np.array_equal(got, want) and m == np.float32(2.0 ** -46)


def test_the_largest_finite_maximum_stays_in_range():
    p = np.zeros(256, np.float32)
    p[::32] = np.finfo(np.float32).max
    _, _, (b0, b1, b2) = unit_of(p)
    z = 65536 * b2 + 256 * b1 + b0
    assert np.abs(z).max() < 2 ** 22 and np.abs(A * z).max() <= 128 * Q_MAX * (1 + 2.0 ** -20)


def test_a_unit_that_takes_the_error_of_the_reciprocal():
    # an approximate reciprocal (1 + d) / m, |d| <= 2^-23, and the unit times 2 - m * inv (fused): half an integer stays half an integer
    for seed in range(1, 40):
        p = products(seed)
        m = np.float32(np.abs(p).max())
        for steps in (-1, 0, 1):
            inv = np.float32(1) / m
            inv = np.nextafter(inv, np.float32(np.inf if steps > 0 else 0)) if steps else inv
            scale = (np.float32(Q_MAX) * inv * np.where(J == 7, np.float32(-1), np.float32(2.0) ** (7 - J)).astype(np.float32))
            z = np.rint(p.astype(np.float64) * scale.astype(np.float64))
            assert np.abs(z).max() < 2 ** 22
            factor = np.float32(2.0 - np.float64(m) * np.float64(inv))
            unit = m * np.float32(1.0 / (128 * Q_MAX)) * factor
            assert np.abs(A * z * np.float64(unit) - p).max() <= np.abs(p).max() * (64 / (128 * Q_MAX) + 2.0 ** -21)


def test_the_unit_times_the_scale_of_the_integers_is_one():
    # The reciprocal moved by up to 2^-17 of itself: the unit that takes 2 - m * inv makes up for it to five roundings of 2^-24 (unit's constant and product,
    # scale, factor, their product); without the factor, or with the error's sign the other way, it does not.
    def worst(factor_of):
        most = 0.0
        for seed in range(1, 40):
            m = np.float32(np.abs(products(seed)).max())
            for steps in (-64, -9, -1, 0, 1, 9, 64):
                inv = np.float32(1) / m
                inv = np.float32(inv + steps * np.spacing(inv))
                factor = np.float32(factor_of(np.float64(m) * np.float64(inv)))
                unit = np.float32(m * np.float32(1.0 / (128 * Q_MAX))) * factor
                scale = np.float32(Q_MAX) * inv
                most = max(most, abs(np.float64(unit) * np.float64(scale) * 128 - 1))
        return most
    five_roundings = 5 * 2.0 ** -24 + 2.0 ** -33       # (the square of the largest error beside them)
    assert worst(lambda m_inv: 2.0 - m_inv) <= five_roundings
    assert worst(lambda m_inv: 1.0) > 8 * five_roundings
    assert worst(lambda m_inv: m_inv) > 16 * five_roundings


def test_reciprocals_above_2_to_126_are_subnormal():
    # flushed to zero by the approximate reciprocal; maxima from 1e37 on are scaled by 2^-64 first, with the same integers
    tiny = np.finfo(np.float32).tiny
    above = np.nextafter(np.float32(2.0 ** 126), np.float32(np.inf))
    assert 0 < np.float32(1) / above < tiny <= np.float32(1) / np.float32(2.0 ** 126) and np.float32(1e37) < above
    p = (products(3) / np.abs(products(3)).max()).astype(np.float32)
    want, _ = words_of(p)
    got, m = words_of((p * np.float32(2.0 ** 127)) * np.float32(2.0 ** -64))
    assert np.array_equal(got, want) and m == np.float32(2.0 ** 63)
