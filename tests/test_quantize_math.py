"""CPU proof (numpy, exhaustive over significand pairs) of the arithmetic with which the fused quantizers avoid dividing:
one multiplication by a rounded-up reciprocal stands in for x / smooth, one for amax / 6 and one for x / scale, and every
decision (scale byte, code) still comes out as the IEEE quotients give it.  Restates qmath::smooth_reciprocal,
qmath::scale_byte_near and qmath::group_codes of svdquant_kernels_b200/csrc/quantize_math.cuh."""
import numpy as np

from oracle import nvfp4_oracle as O

f32, f64 = np.float32, np.float64
NUDGE = 1.0 + 2.0 ** -22
SIXTH = f32((1.0 / 6.0) * (1.0 - 2.0 ** -22))


def _reciprocal(s):
    """the table entry: RN((1 / s)(1 + 2^-22)); float64 carries the value to 2^-52"""
    return f32((1.0 / f64(s)) * NUDGE)


def _scale_byte_near(f):
    v = (f.astype(f32) * SIXTH).astype(f32)
    snapped = ((v.view(np.uint32) + np.uint32(8)) & np.uint32(0xFFFFFFF0)).view(f32)
    return O.e4m3_encode(np.minimum(snapped, f32(448.0)))


def _scale_byte_exact(q):
    s = np.minimum(np.maximum((q / f32(6.0)).astype(f32), f32(1e-12)), f32(448.0))
    return O.e4m3_encode(s)


def test_scale_byte_of_the_near_quotient_equals_that_of_the_ieee_quotient():
    """Every pair of 11-bit significands (fp16; bf16 has fewer bits), quotients in every binade of the e4m3 range,
    subnormals and the clamp included; and the same for a quotient that is exact (no smoothing, or __fdiv_rn)."""
    x = np.arange(1024, 2048, dtype=f32)
    for ms in range(1024, 2048):
        s = f32(ms)
        q1 = (x / s).astype(f32)
        f1 = (x * _reciprocal(s)).astype(f32)
        # binades of amax / 6 from below the smallest scale (2^-10 is its rounding bound) to above 448
        exps = range(-10, 13) if ms % 16 == 0 or ms in (1025, 2047) else (-8, -6, -4, -1, 11)
        for e in exps:
            k = f32(2.0 ** e)
            want = _scale_byte_exact(q1 * k)
            assert (_scale_byte_near(f1 * k) == want).all(), (ms, e)
            assert (_scale_byte_near(q1 * k) == want).all(), (ms, e)


def test_codes_from_the_near_quotient_equal_the_ieee_ones():
    """Codes of x / s against every scale significand J (1..15), for every pair of 11-bit significands and all ratios up
    to past saturation: the E2M1 conversion (nearest; the kernel's hardware conversion) of f c lands on the side of
    each bound where the exact quotient is, a quotient on a bound counting as above it.  c is the approximate
    reciprocal of the scale (at most one unit off) times (1 + 2^-21): both ends of that range are tried."""
    bounds = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])
    x = np.arange(1024, 2048, dtype=f64)
    step = 7                                        # every 7th divisor, all residues over the run of exponents
    for ms in list(range(1024, 2048, step)) + [1025, 1365, 2046, 2047]:
        s = f64(ms)
        f1 = (x.astype(f32) * _reciprocal(f32(ms))).astype(f32)
        for J in range(1, 16):
            r = f32(1.0 / J)
            for rc in (np.nextafter(r, f32(0)), r, np.nextafter(r, f32(2))):
                c = f32(rc * f32(1.0 + 2.0 ** -21))
                for e in range(-3, 8):
                    k = 2.0 ** e
                    ratio_max = 2.0 * k / J
                    if ratio_max < 0.2 or k / (2 * J) > 12:
                        continue
                    w = (f1 * f32(k) * c).astype(f32).astype(f64)
                    got = (w[:, None] > bounds).sum(1)
                    assert not np.isin(w, bounds).any()
                    # exact: x k / (s J) >= b  <=>  4 x k >= 4 b s J, all integers times powers of two below 2^53
                    want = (4.0 * k * x[:, None] >= 4.0 * bounds * s * J).sum(1)
                    assert (got == want).all(), (ms, J, e)


def test_exact_quotients_and_zeros():
    """Without smoothing (f = x) the same multiplications decide correctly, and a -0 input loses its sign in f = x r + 0."""
    bounds = np.array([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])
    x = np.arange(1, 2048, dtype=f64)
    for J in range(1, 16):
        for rc in (np.nextafter(f32(1.0 / J), f32(0)), f32(1.0 / J), np.nextafter(f32(1.0 / J), f32(2))):
            c = f32(rc * f32(1.0 + 2.0 ** -21))
            for e in range(-14, 5):
                w = (x.astype(f32) * f32(2.0 ** e) * c).astype(f32).astype(f64)
                assert ((w[:, None] > bounds).sum(1) == (4.0 * 2.0 ** e * x[:, None] >= 4.0 * bounds * J).sum(1)).all(), (J, e)
    assert not np.signbit(f32(-0.0) * f32(3.0) + f32(0.0))
