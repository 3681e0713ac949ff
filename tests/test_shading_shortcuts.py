"""The integer division of the sampler's digit groups and the plain cases of
sphere_lambert, restated with numpy, against their definitions (CPU)."""
import numpy as np
import pytest

F = np.float32


def halton_bases():
    """(base, pow_base) of the sampler's dimensions after the first: the
    largest power of the prime at most 500."""
    primes = [p for p in range(3, 1620) if all(p % d for d in range(2, int(p ** 0.5) + 1))][:255]
    out = []
    for b in primes:
        pb = b
        while pb * b <= 500:
            pb *= b
        out.append(pb)
    return out


@pytest.mark.parametrize("part", range(4))
def test_digit_group_division(part):
    for pb in sorted(set(halton_bases()))[part::4]:
        check_division(pb)


def check_division(pb):
    rng = np.random.default_rng(pb)
    top = (1 << 32) - 1
    edge = [k * pb + e for k in (0, 1, 2, top // pb - 1, top // pb) for e in (-1, 0, 1)] + [top, top - 1, 1 << 31]
    q = np.array([v for v in edge if 0 <= v <= top] + list(rng.integers(0, 1 << 32, 4096)), np.uint64)
    t = (q * np.uint64((1 << 32) // pb)) >> np.uint64(32)
    r = q - t * np.uint64(pb)
    low = r >= pb
    t, r = np.where(low, t + np.uint64(1), t), np.where(low, r - np.uint64(pb), r)
    assert np.array_equal(t, q // np.uint64(pb)) and np.array_equal(r, q % np.uint64(pb))


def test_one_minus_a_float_in_double_or_float():
    rng = np.random.default_rng(3)
    x = rng.integers(0, 1 << 32, 4000000, dtype=np.uint64).astype(np.uint32).view(F)
    x = np.concatenate([x[np.isfinite(x)], np.ldexp(F(1.0) + rng.random(200000).astype(F), rng.integers(-60, 61, 200000)).astype(F)])
    with np.errstate(over="ignore"):
        assert np.array_equal((1.0 - x.astype(np.float64)).astype(F), F(1.0) - x)


@pytest.mark.parametrize("near", [0.0, 0.9, 0.999, 0.9999999])
def test_sphere_lambert_plain_cases(near):
    """Where the cosine test takes a plain case, the angle test of the full
    form does too, by far more than an arc cosine's rounding."""
    rng = np.random.default_rng(int(near * 1e7))
    rcos = (near + (1.0 - near) * rng.random(200000)).astype(F)
    rcos = np.minimum(rcos, F(1.0))
    nlcos = rng.uniform(-1.0, 1.0, rcos.size).astype(F)
    # half of them around the horizon's edges
    s = np.sqrt(np.maximum(1.0 - rcos.astype(np.float64) ** 2, 0.0))
    k = rcos.size // 2
    nlcos[:k] = np.clip(np.sign(nlcos[:k]) * s[:k] + rng.normal(0.0, 3e-3, k), -1.0, 1.0).astype(F)
    rsin2 = (1.0 - (rcos * rcos).astype(np.float64)).astype(F)
    assert np.array_equal(rsin2, F(1.0) - rcos * rcos)  # the kernels subtract in 32 bits
    m = F(1e-3)
    inner, outer = np.abs(nlcos) + m, np.abs(nlcos) - m
    whole = (outer > 0) & (outer * outer > rsin2)
    above, below = whole & (nlcos > 0), whole & (nlcos < 0)
    nl, r = np.arccos(nlcos.astype(np.float64)), np.arccos(rcos.astype(np.float64))
    cut = (outer > 0) & ~whole & (inner * inner < rsin2)
    mostly_above, mostly_below = cut & (nlcos > 0), cut & (nlcos < 0)
    assert above.sum() > 1000 and below.sum() > 1000
    for mostly, lo, hi in ((mostly_above, np.pi / 2 - r, np.pi / 2 + 0 * r), (mostly_below, np.pi / 2 + 0 * r, np.pi / 2 + r)):
        assert mostly.sum() > 1000 or near > 0.999
        assert np.all(nl[mostly] > lo[mostly] + 1e-4) and np.all(nl[mostly] < hi[mostly] - 1e-4)
    assert np.all(nl[above] < np.pi / 2 - r[above] - 1e-4)
    assert np.all(nl[below] > np.pi / 2 + r[below] + 1e-4)
