"""The sampler's division and the light estimate's quick cases: the kernels'
own functions (shade_math.h, compiled for the host) against the forms that
they stand for, bit for bit (CPU)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "psychopath_cpp_b200", "csrc")
F = np.float32


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("shade") / "libshade_host.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-fPIC", "-shared", "-I" + CSRC,
                    os.path.join(HERE, "shade_host.cpp"), "-o", so, "-lm"], check=True)
    return C.CDLL(so)


def p(a):
    return a.ctypes.data_as(C.c_void_p)


def divisors():
    """The sampler's digit groups: of each prime base the largest power up to
    500."""
    primes = [b for b in range(3, 1620) if all(b % d for d in range(2, int(b ** 0.5) + 1))][:255]
    return sorted({b ** max(1, int(np.log(500) / np.log(b) + 1e-9)) for b in primes})


@pytest.mark.parametrize("part", range(4))
def test_division(lib, part):
    top = (1 << 32) - 1
    for d in divisors()[part::4]:
        edges = [k * d + e for k in (0, 1, 2, top // d - 1, top // d) for e in (-1, 0, 1)] + [top - 1, top, 1 << 31]
        x = np.concatenate([np.array([v for v in edges if 0 <= v <= top], np.uint32),
                            np.random.default_rng(d).integers(0, 1 << 32, 4096, dtype=np.uint64).astype(np.uint32)])
        q, r = np.empty_like(x), np.empty_like(x)
        lib.divisions(x.size, p(x), C.c_uint32(d), p(q), p(r))
        assert np.array_equal(q, x // np.uint32(d)) and np.array_equal(r, x % np.uint32(d))


@pytest.mark.parametrize("near", [0.0, 0.9, 0.999, 0.9999999])
def test_sphere_lambert(lib, near):
    rng = np.random.default_rng(int(near * 1e7))
    n = 400000
    rcos = np.minimum((near + (1.0 - near) * rng.random(n)).astype(F), F(1.0))
    nlcos = rng.uniform(-1.0, 1.0, n).astype(F)
    # half of them around the limits: the cap's rim on the horizon, its centre
    # on the horizon, and the normal's own direction, past 1 by rounding
    s = np.sqrt(np.maximum(1.0 - rcos.astype(np.float64) ** 2, 0.0))
    k, m = n // 2, n // 8
    nlcos[:k] = (np.sign(nlcos[:k]) * s[:k] + rng.normal(0.0, 2e-3, k)).astype(F)
    nlcos[:m] = rng.normal(0.0, 1e-3, m).astype(F)
    nlcos[m:2 * m] = F(1.0) + (rng.integers(-4, 5, m) * 2.0 ** -23).astype(F)
    nlcos[2 * m:3 * m] = F(-1.0) + (rng.integers(-4, 5, m) * 2.0 ** -23).astype(F)
    got, want, cut = np.empty(n, F), np.empty(n, F), np.empty(n, np.int32)
    lib.lambert(n, p(nlcos), p(rcos), p(got), p(cut))
    lib.lambert_plain(n, p(nlcos), p(rcos), p(want))
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    # a cap whose cosine is not a number has none of the cases; -0 and +0 weigh
    # the same
    assert np.all(same | ((got == 0.0) & (want == 0.0)))
    assert (cut < 0).sum() > n // 20 and (cut >= 0).sum() > n // 20


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 9, 17])
def test_a_time_s_place_lies_within_the_samples(lib, count):
    rng = np.random.default_rng(count)
    t = rng.integers(0, 1 << 32, 200000, dtype=np.uint64).astype(np.uint32).view(F)
    t = np.concatenate([t, rng.uniform(-3.0, 2.0, 200000).astype(F), np.array([0.0, -0.0, 1.0, np.nextafter(F(1), F(0)),
                                                                               np.inf, -np.inf, np.nan], F)])
    first, last, alpha = np.empty(t.size, np.int32), np.empty(t.size, np.int32), np.empty(t.size, F)
    lib.positions(t.size, p(t), count, p(first), p(last), p(alpha))
    assert first.min() == 0 and last.max() == count - 1 and np.all(first <= last)
    inside = (t >= 0) & (t < 1)
    at = t[inside] * F(count - 1)
    assert np.array_equal(first[inside], at.astype(np.int32)) and np.array_equal(alpha[inside], at - at.astype(np.int32))
