"""The tile decode divides by trunc((x + 0.5) * rcp(n)) in FP32 (small_div in gsv_bin.cu), for dividends up to four
million: exact at the multiples of every divisor and beside them, where it could fail first."""
import numpy as np

F = np.float32
LIMIT = 4_000_000


def _small_div(x, n):
    return ((x.astype(F) + F(0.5)) * (F(1) / n.astype(F))).astype(np.int32)


def _check(x, n):
    keep = (x >= 0) & (x < LIMIT)
    x, n = x[keep], n[keep]
    assert np.array_equal(_small_div(x, n), x // n)


def test_near_multiples():
    n = np.arange(1, 65536, dtype=np.int64)  # at most 65535 tiles on an axis
    top = LIMIT // n
    for k in (1, 2, 3, top // 3, top // 2, top - 1, top):
        for d in (-1, 0, 1):
            _check(k * n + d, n)


def test_every_dividend_of_some_divisors():
    x = np.arange(LIMIT, dtype=np.int64)
    for n in (1, 2, 3, 5, 7, 37, 641, 4093, 18432, 65521, 65535):
        _check(x, np.full_like(x, n))
