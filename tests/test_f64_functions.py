"""The f64 functions of csrc/sb_f64.cuh and csrc/sb_line.cuh on the GPU, over their ranges and at their ends: zeros,
subnormals, the ends of the FP32 range, infinities, no numbers.

Bounds: conversions bit for bit. Reciprocal, square root and its reciprocal: 2 units in the last place (a third-order
step's error below 2^-63 and the roundings of its last operations). The exponential: 2 units (table entry, series
product, last addition, each half of one, and 4e-18 of the series). x^p: the exponent p log2 x is rounded in f64 (2^-53 of
its size, twice) and log2 x of the rest has an error of some 2^-52, which p multiplies: 2^-52 (|p ln x| + 2 p + 4).
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.join(HERE, "..")
ENDS = np.array([0.0, 5e-324, 2.0**-1030, 2.0**-1022, 2.0**-700, 2.0**-150, 2.0**-149, 1.5 * 2.0**-149, 2.0**-140, 2.0**-127,
                 np.nextafter(2.0**-126, 0), 2.0**-126, 2.0**-101, 2.0**-100, 1e-20, 0.1, 1.0, 1.0 - 2.0**-53, 1.0 + 2.0**-24, 3.0,
                 np.nextafter(2.0**100, 0), 2.0**100, np.nextafter(2.0**127, 0), 2.0**127, 3.4028234663852886e38,
                 3.4028235677973366e38, 1e39, 2.0**700, 1.7e308, np.inf, np.nan])


@pytest.fixture(scope="module")
def device(gpu_lib, tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("f64") / "f64_functions_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "stormbird_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(HERE, "f64_functions_check.cu"), "-o", exe], check=True, capture_output=True)

    def call(name, *args):
        data = np.stack(np.broadcast_arrays(*[np.asarray(a, dtype=np.float64) for a in args]), axis=-1)
        out = subprocess.run([exe, name], input=data.tobytes(), capture_output=True, check=True, timeout=120).stdout
        return np.frombuffer(out, dtype=np.float64)

    return call


def values(lo, hi, n=100_000):
    rng = np.random.default_rng(7)
    return np.concatenate([ENDS, -ENDS, np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)])


def same(a, b):
    """Bit for bit, every no number the same."""
    both = np.isnan(a) & np.isnan(b)
    return np.array_equal(a[~both].view(np.uint64), b[~both].view(np.uint64))


@pytest.mark.parametrize("name", ["to_f32_rn", "to_f64_exact"])
def test_conversions(device, name):
    v = values(-160, 130)
    with np.errstate(over="ignore"):
        f = v.astype(np.float32)
    assert same(device(name, v), f.astype(np.float64))


def test_to_f32(device):
    """Ties away from zero in its range, 0 below it; from 2^128 up 0 as well, which callers rule out."""
    v = values(-160, 130)
    out, mag = device("to_f32", v), np.abs(v)
    with np.errstate(over="ignore", invalid="ignore"):
        inside = (mag >= 2.0**-126) & (mag < 2.0**128)
        even = v.astype(np.float32)
        away = np.nextafter(even, np.copysign(np.float32(np.inf), v).astype(np.float32))
        tie = np.abs(v - even.astype(np.float64)) == np.abs(away.astype(np.float64) - v)
    want = np.where(tie, away, even).astype(np.float64)
    assert np.array_equal(out[inside], want[inside])
    assert np.all(out[~inside] == 0.0)


@pytest.mark.parametrize("name", ["rcp", "sqrt", "rsqrt"])
def test_roots(device, name):
    v = values(-1074, 1023)
    out = device(name, v)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        want = {"rcp": lambda: 1.0 / v, "sqrt": lambda: np.sqrt(v), "rsqrt": lambda: 1.0 / np.sqrt(v)}[name]()
    fine = np.isfinite(want) & (want != 0.0)
    assert same(out[~fine], want[~fine])
    assert np.max(np.abs(out[fine] - want[fine]) / np.spacing(np.abs(want[fine]))) <= 2.0


def test_exp2(device):
    """2^((n + f) / 512) wherever the result is a normal number."""
    rng = np.random.default_rng(11)
    n = np.concatenate([[-512 * 1021, -512 * 960, -512 * 900, -1, 0, 511, 512, 512 * 99, 512 * 1022],
                        rng.integers(-512 * 1021, 512 * 1022, 50_000)]).astype(np.float64)
    f = rng.uniform(-0.6, 0.6, len(n))
    whole = np.floor(n / 512)
    part = (n - 512 * whole).astype(np.longdouble) + f  # exact to 2^-63 of 512
    want = np.exp2(part / 512)                           # [1, 2), scaled exactly
    out = np.ldexp(device("exp2", n, f), -whole.astype(int))
    assert np.max(np.abs((out - want).astype(np.float64))) <= 2.0 * 2.0**-52


def test_pow(device):
    rng = np.random.default_rng(12)
    x = np.concatenate([[0.0, 1.0, 1.0 - 2.0**-53, 2.0**-60, 2.0**-60 * 1.999, 2.0**-61, 1e-300, 1e-305, 0.5, 2.0**-0.5],
                        2.0 ** rng.uniform(-62, 0, 20_000)])
    for p in (0.0, 0.5, 1.0, 1.6, 2.0, 7.3, 16.0, 16.5, -1.0):
        out = device("pow", x, p)
        with np.errstate(divide="ignore", under="ignore"):
            want = np.power(x.astype(np.longdouble), np.longdouble(p))
            log = np.abs(p * np.log(np.maximum(x, 5e-324)))
            rounded = want.astype(np.float64)
        ends = (rounded == 0.0) | np.isinf(rounded)
        assert same(out[ends], rounded[ends])
        fine = ~ends & (rounded >= 2.0**-1022)  # (subnormal results are the library function's)
        err = np.abs((out[fine].astype(np.longdouble) / want[fine] - 1).astype(np.float64))
        assert np.all(err <= 2.0**-52 * (log[fine] + 2.0 * p + 4.0) if p >= 0 else err <= 2.0**-50)
