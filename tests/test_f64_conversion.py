"""The integer-pipe conversions of the panel records (f64_to_f32_rn, f32_to_f64_exact in csrc/sb_f64.cuh),
restated on the host: bit for bit the conversions they stand in for, at ties, at the ends of the normal
range (beyond it they call the conversion), at zeros and at random."""
import numpy as np

U = np.uint64


def to_f32(v):
    """f64_to_f32_rn for values it does not hand on, and whether it hands them on."""
    bits = v.view(np.uint64)
    hi, lo = (bits >> U(32)).astype(np.uint64), (bits & U(0xFFFFFFFF)).astype(np.uint64)
    mag = ((hi & U(0x7FFFFFFF)) - U(0x38000000)) & U(0xFFFFFFFF)
    outside = ((mag - U(0x00100000)) & U(0xFFFFFFFF)) >= U(0x0FE00000)
    zero = ((hi & U(0x7FFFFFFF)) | lo) == 0
    out = ((mag << U(3)) | (lo >> U(29))) & U(0xFFFFFFFF)
    out = out + (((lo & U(0x1FFFFFFF)) + U(0x0FFFFFFF) + (out & U(1))) >> U(29))
    out = np.where(zero, hi, out | (hi & U(0x80000000)))
    return out.astype(np.uint32).view(np.float32), outside & ~zero


def to_f64(v):
    u = v.view(np.uint32).astype(np.uint64)
    mag = u & U(0x7FFFFFFF)
    outside = ((mag - U(0x00800000)) & U(0xFFFFFFFF)) >= U(0x7F000000)
    hi = np.where(mag == 0, u, ((mag >> U(3)) + U(0x38000000)) | (u & U(0x80000000)))
    lo = np.where(mag == 0, U(0), (u << U(29)) & U(0xFFFFFFFF))
    return ((hi << U(32)) | lo).view(np.float64), outside & (mag != 0)


def samples():
    rng = np.random.default_rng(3)
    v = rng.normal(size=200_000) * 10.0 ** rng.uniform(-36, 36, 200_000)
    f = rng.integers(0x00800000, 0x7F000000, 50_000).astype(np.uint32).view(np.float32).astype(np.float64)
    up = np.nextafter(f.astype(np.float32), np.float32(np.inf)).astype(np.float64)
    ties = 0.5 * (f + up)  # halfway between neighbouring floats, and a bit to each side
    edge = np.array([0.0, -0.0, 2.0**-126, np.nextafter(2.0**-126, 0), 2.0**-150, 5e-324, 2.0**127, np.nextafter(2.0**127, 0),
                     3.4028235677973366e38, 1e300, np.inf, -np.inf, 1.0, 0.5, 1.0 - 2.0**-53, 1.0 + 2.0**-24])
    return np.concatenate([v, f, ties, np.nextafter(ties, 0), np.nextafter(ties, np.inf), edge, -edge])


def test_to_f32():
    v = samples()
    ours, handed_on = to_f32(v)
    with np.errstate(over="ignore"):
        ref = v.astype(np.float32)
    ok = ~handed_on
    assert np.array_equal(ours[ok].view(np.uint32), ref[ok].view(np.uint32))
    big = (np.abs(v) >= 2.0**-126) & (np.abs(v) < 2.0**127)
    assert not np.any(handed_on & big)  # the whole range it is made for


def test_to_f64():
    with np.errstate(over="ignore"):
        f = samples().astype(np.float32)
    ours, handed_on = to_f64(f)
    ok = ~handed_on
    assert np.array_equal(ours[ok].view(np.uint64), f.astype(np.float64)[ok].view(np.uint64))
    assert not np.any(handed_on & np.isfinite(f) & (np.abs(f) >= 2.0**-126))
