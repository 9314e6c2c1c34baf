"""Division by a host-known divisor as a high multiply, an add and a shift (the kernels' item -> pixel maps):
exact for every n < 2^31, and the sum stays below 2^32."""
import numpy as np


def fast_div(d):
    s = 0
    while s < 31 and (1 << s) < d:
        s += 1
    return s, ((((1 << s) - d) << 32) // d + 1) & 0xFFFFFFFF


def test_quotients_are_exact():
    rng = np.random.default_rng(1)
    divisors = sorted(set(list(range(1, 70)) + [2 ** k + e for k in range(1, 31) for e in (-1, 0, 1) if 2 ** k + e > 0] +
                          [int(x) for x in 2.0 ** rng.uniform(0, 31, 200)]))
    for d in divisors:
        s, m = fast_div(d)
        k = rng.integers(0, (2 ** 31 - 1) // d + 1, 500, dtype=np.uint64) * np.uint64(d)
        n = np.unique(np.concatenate([k, k + np.uint64(d - 1), k + np.uint64(1), np.maximum(k, np.uint64(1)) - np.uint64(1),
                                      np.array([0, 1, 2 ** 31 - 1], dtype=np.uint64)]))
        n = n[n < 2 ** 31]
        t = ((np.uint64(m) * n) >> np.uint64(32)) + n
        assert t.max() < 2 ** 32
        np.testing.assert_array_equal(t >> np.uint64(s), n // np.uint64(d))
