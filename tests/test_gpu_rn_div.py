"""The quotients of rn_div.cuh against the compiler's division, over seeded random
operands of the domain the header states: with a good guard div equals `/` for
dividends that are zero or at least 2^-900 (FP32: 2^-90) in magnitude; quotient_mag
falls back by itself and takes divisors of either sign; sixth and third take any
value. Equal means every bit, a zero's sign apart for quotient_mag."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from scale_b200 import build

pytestmark = pytest.mark.gpu

N = 1 << 21
# least dividend's, greatest dividend's and divisors' binary exponents
RANGE = {np.float64: (-900, 1000, -1015, 1020), np.float32: (-90, 120, -120, 126)}


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = tmp_path_factory.mktemp("rn") / "rn_div_probe.so"
    src = Path(__file__).with_name("rn_div_probe.cu")
    subprocess.run([build._nvcc(), "-O3", "-std=c++17", *build.ARCH, "-ccbin", build._host_cxx(), "-I", str(build.CSRC),
                    "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared", "-o", str(out), str(src)], check=True)
    return C.CDLL(str(out))


def _random(rng, t, lo, hi, signed=True):
    x = (1.0 + rng.random(N)).astype(np.float64)
    if t is np.float32:
        x = x.astype(t).astype(np.float64)
        x[x >= 2.0] = 1.0
    x = np.ldexp(x, rng.integers(lo, hi, N))
    return (x * np.where(rng.random(N) < 0.5, -1.0, 1.0) if signed else x).astype(t)


def _call(probe, what, a, b):
    import torch

    t = a.dtype.type
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b, np.zeros(a.size, t), np.zeros(a.size, t))]
    ok = torch.zeros(a.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rc = probe.rn_probe(int(t is np.float64), what, *(C.c_void_p(x.data_ptr()) for x in dev), C.c_void_p(ok.data_ptr()),
                        C.c_size_t(a.size))
    assert rc == 0
    return dev[2].cpu().numpy(), dev[3].cpu().numpy(), ok.cpu().numpy().astype(bool)


def _bits(x):
    return x.view(np.int64 if x.dtype == np.float64 else np.int32)


@pytest.mark.parametrize("t", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("what", [0, 1], ids=["div", "shared_reciprocal"])
def test_div_with_a_good_guard(gpu, probe, t, what):
    rng = np.random.Generator(np.random.PCG64(11))
    alo, ahi, blo, bhi = RANGE[t]
    a, b = _random(rng, t, alo, ahi), _random(rng, t, blo, bhi, signed=False)
    # half of the pairs at ordinary sizes, where no quotient overflows
    a[: N // 2], b[: N // 2] = _random(rng, t, -40, 40)[: N // 2], _random(rng, t, -40, 40, signed=False)[: N // 2]
    a[::1000] = t(0.0)
    got, want, ok = _call(probe, what, a, b)
    assert ok[: N // 2].all()
    assert np.array_equal(_bits(got)[ok], _bits(want)[ok])
    assert np.isfinite(want[ok]).all()


@pytest.mark.parametrize("t", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("what", [0, 1], ids=["div", "shared_reciprocal"])
def test_guard_refuses_what_the_method_cannot_form(gpu, probe, t, what):
    tiny, huge = np.finfo(t).smallest_subnormal, np.finfo(t).max
    a = np.array([1.0, 1.0, 1.0, 1.0, 1.0, np.inf, np.nan, huge, 0.0], t)
    b = np.array([0.0, np.inf, np.nan, -2.0, tiny, 1.0, 1.0, 0.25, 0.0], t)
    ok = _call(probe, what, a, b)[2]
    assert not ok.any()


@pytest.mark.parametrize("t", [np.float64, np.float32], ids=["fp64", "fp32"])
def test_quotient_mag(gpu, probe, t):
    rng = np.random.Generator(np.random.PCG64(12))
    alo, ahi, blo, bhi = RANGE[t]
    a, b = _random(rng, t, alo, ahi), _random(rng, t, blo, bhi)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -3.0, np.finfo(t).max, np.finfo(t).tiny], t)
    n = special.size
    a[: n * n], b[: n * n] = np.repeat(special, n), np.tile(special, n)
    # (a tiny dividend by a huge divisor: the domain the header states starts above it)
    skip = (np.abs(a) < np.ldexp(t(1.0), alo)) & (a != 0)
    got, want, _ = _call(probe, 2, a, b)
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    assert same[~skip].all()


@pytest.mark.parametrize("t", [np.float64, np.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("what", [3, 4], ids=["sixth", "third"])
def test_constant_divisors(gpu, probe, t, what):
    rng = np.random.Generator(np.random.PCG64(13))
    info = np.finfo(t)
    a = _random(rng, t, info.minexp - info.nmant, info.maxexp)
    a[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, info.max, info.smallest_subnormal, info.tiny]
    got, want, _ = _call(probe, what, a, a)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(_bits(got)[~nan], _bits(want)[~nan])
