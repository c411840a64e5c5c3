"""CPU proof (numpy, over every pair of 11-bit significands) of the arithmetic with which the fused quantizers avoid
dividing: one multiplication by a rounded-up reciprocal stands in for x / smooth, one for amax / 6 and one for x / scale,
and every decision (scale byte, code) still comes out as the IEEE quotients give it.  Restates qmath::smooth_reciprocal,
qmath::scale_byte_near and qmath::quantize_group_near of svdquant_kernels_b200/csrc/quantize_math.cuh.

fp16 significands have 11 bits, bf16's fewer.  Powers of two pass through every multiplication here unchanged (the kernels
leave this path where something could over- or underflow), so one binade of x against one of smooth stands for all."""
import numpy as np

from oracle import nvfp4_oracle as O

f32, f64 = np.float32, np.float64
NUDGE = 1.0 + 2.0 ** -22
SIXTH = f32((1.0 / 6.0) * (1.0 - 2.0 ** -22))
SIG = np.arange(1024, 2048, dtype=f64)               # every 11-bit significand
X, S = SIG[None, :], SIG[:, None]


def _near():
    """f = x r for every pair [smooth, x]; float64 carries the table entry's value to 2^-52"""
    r = ((1.0 / S) * NUDGE).astype(f32)
    return (X.astype(f32) * r).astype(f32)


def _snapped(f):
    """the near scale of qmath::scale_byte_near, before its conversion to E4M3"""
    v = (f.astype(f32) * SIXTH).astype(f32)
    return ((v.view(np.uint32) + np.uint32(8)) & np.uint32(0xFFFFFFF0)).view(f32)


def test_near_quotients_lie_in_the_window():
    """Above the exact quotient by 2^-24 to 2^-21.4 of it."""
    rel = _near().astype(f64) / (X / S) - 1.0         # good to 2^-52
    assert rel.min() >= 2.0 ** -24 and rel.max() <= 2.0 ** -21.4


def test_scale_byte_of_the_near_quotient_equals_that_of_the_ieee_quotient():
    """In every binade of the e4m3 range, subnormals, the clamp and what lies below and above included.  The largest near
    quotient of a group may be another element's than the largest quotient; it still lies in the window above that one,
    so the window's ends are tried beside the near quotient itself.  So is the IEEE quotient (no smoothing, or __fdiv_rn)."""
    q = (X / S).astype(f32)                           # numpy divides correctly rounded; 11 by 11 bits: rounded once
    assert (q == (X.astype(f32) / S.astype(f32)).astype(f32)).all()
    low = np.nextafter((X / S * (1.0 + 2.0 ** -24)).astype(f32), f32(0))
    low = np.where(low.astype(f64) < X / S, np.nextafter(low, f32(4)), low)
    high = (X / S * (1.0 + 2.0 ** -21.4)).astype(f32)
    want6 = (q / f32(6.0)).astype(f32)
    tried = [_snapped(f) for f in (_near(), low, high, q)]
    for e in range(-10, 13):                          # amax / 6 from below 2^-10, the smallest scale's bound, to above 448
        k = f32(2.0 ** e)
        want = O.e4m3_encode(np.minimum(np.maximum(want6 * k, f32(1e-12)), f32(448.0)))
        for near in tried:
            assert (O.e4m3_encode(np.minimum(near * k, f32(448.0))) == want).all(), e


def test_codes_from_the_near_quotient_equal_the_ieee_ones():
    """Codes of x / s against every scale significand J (1..15): the E2M1 conversion (nearest; the kernel's hardware
    conversion) of f c lands on the side of each bound where the exact quotient is, a quotient on a bound counting as above
    it, and never on the bound itself.  c is the approximate reciprocal of the scale (at most one unit off) times
    (1 + 2^-21): both ends of that range are tried.  The bounds are 1, 1.25, 1.5 and 1.75 times powers of two."""
    f = _near()
    for J in range(1, 16):
        r = f32(1.0 / J)
        near = [(f * f32(rc * f32(1.0 + 2.0 ** -21))).astype(f32) for rc in (np.nextafter(r, f32(0)), r, np.nextafter(r, f32(2)))]
        lowest, highest = min(w.min() for w in near), max(w.max() for w in near)
        for e in range(-6, 3):
            for sig in (1.0, 1.25, 1.5, 1.75):
                bound = sig * 2.0 ** e
                if not lowest * 0.5 < bound < highest * 2.0:
                    continue
                above = X >= bound * J * S            # exact: both sides are integers times powers of two below 2^53
                for w in near:
                    assert ((w > f32(bound)) == above).all() and not (w == f32(bound)).any(), (J, bound)


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
