"""The FP32 block CG's alpha is the FP64 quotient rounded to FP32, also where that
quotient lies within 2^-49 (relative) of the middle of two FP32 values: one step on
a diagonal operator whose sums r^T r = R and p^T w = Q are exact, with R / Q a hair
above such a middle.  No tolerance: the coefficient is known exactly."""
from math import isqrt

import numpy as np
import pytest

from gcge_gb300 import problems as P

pytestmark = pytest.mark.gpu

PARTS = 8  # squares a sum is written with


def squares(total, most):
    """Eight integers up to `most` whose squares add up to `total`."""
    parts, rest = [], total
    for _ in range(4):
        parts.append(isqrt(total // PARTS))
        rest -= parts[-1] ** 2
    for x in range(isqrt(rest // 4), 0, -1):
        r3 = rest - x * x
        for y in range(isqrt(r3 // 3), max(isqrt(r3 // 3) - 40, 0), -1):
            r2 = r3 - y * y
            for z in range(isqrt(r2 // 2), max(isqrt(r2 // 2) - 400, 0), -1):
                w = isqrt(r2 - z * z)
                if w * w == r2 - z * z and max(x, y, z, w) <= most:
                    return parts + [x, y, z, w]
    return None


def quotients(count):
    """(R, Q, the FP32 value of R / Q): m / 2^25 with m odd is the middle of two FP32
    values in [1/2, 1), and R 2^25 = m Q + 1."""
    rng = np.random.default_rng(7)
    out = []
    while len(out) < count:
        q = int(rng.integers(1 << 24, 1 << 25)) * 2 + 1
        m = (-pow(q, -1, 1 << 25)) % (1 << 25)
        r = (m * q + 1) >> 25
        if m < (1 << 24) or r % 2 == 0:
            continue
        b3 = (q - r) // 2  # R = a + b3, Q = a + 3 b3
        a, b = squares(r - b3, 4095), squares(b3, 2364)
        if a and b:
            out.append((a, b, np.float32((m + 1) / 2.0 ** 25)))
    return out


def test_alpha_is_the_rounded_quotient(gpu_lib):
    k = 40
    cases = quotients(k)
    n = 32 * 2 * PARTS
    d = np.ones(n)
    d[32 * PARTS:] = 3.0
    c = np.zeros((n, k))
    for j, (a, b, _) in enumerate(cases):
        c[0::32, j] = a + b  # one entry a slice: every FP32 sum is exact
    x, it = gpu_lib.block_pcg(P.diag_matrix(d), None, 0.0, c, np.zeros_like(c), max_iter=1,
                              rate=0.0, tol=0.0, fp32=True)
    assert it == 1
    alpha = np.array([al for _, _, al in cases], dtype=np.float32)
    np.testing.assert_array_equal(x, (alpha * c.astype(np.float32)).astype(np.float64))
