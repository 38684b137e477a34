"""The last step of pivot_inv, y <- RN(y + y (1 - x y)), rounds every start within one ulp of 1/x
to RN(1/x), for every significand of x but all ones.

With d = 1 - x y exact and |d| < 2^-52 the sum is (1 - d^2) / x before its rounding, so it rounds
otherwise than 1/x only when a midpoint lies between the two: x = X 2^-52, midpoint M 2^-54 with
M odd, X M = 2^106 - j and 0 < j < d^2 2^106 < 4.  The three numbers are factored here, and the
significands X among their divisors are tried with every start."""
import os
import subprocess
from fractions import Fraction

import pytest

FACTORS = {
    1: [3, 107, 6361, 69431, 20394401, 28059810762433],
    2: [2, 7, 7, 31, 71, 127, 151, 337, 29191, 106681, 122921, 152041],
    3: [2327027, 34864072662073401681969743],
}


def _is_prime(n):
    """Miller-Rabin with the first twenty primes as bases."""
    bases = [2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71]
    if n in bases:
        return True
    if any(n % p == 0 for p in bases):
        return False
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in bases:
        v = pow(a, d, n)
        if v in (1, n - 1):
            continue
        for _ in range(s - 1):
            v = v * v % n
            if v == n - 1:
                break
        else:
            return False
    return True


def _significands():
    """X in (2^52, 2^53) with X M = 2^106 - j, M odd, M in (2^53, 2^54), j = 1, 2, 3."""
    out = []
    for j, primes in FACTORS.items():
        n = (1 << 106) - j
        prod, divisors = 1, {1}
        for p in primes:
            assert _is_prime(p)
            prod *= p
            divisors |= {d * p for d in divisors}
        assert prod == n
        out += [x for x in divisors
                if 1 << 52 < x < 1 << 53 and 1 << 53 < n // x < 1 << 54 and (n // x) % 2]
    return sorted(out)


def _round(v):
    """v in [1/2, 1] to the nearest multiple of 2^-53, ties to even."""
    n, r = divmod(v.numerator << 53, v.denominator)
    twice = 2 * r
    return n + (twice > v.denominator or (twice == v.denominator and n % 2))


def test_last_step_rounds_right():
    ones = (1 << 53) - 1
    xs = _significands()
    assert len(xs) == 33 and ones in xs
    for sig in xs + [(1 << 52) + 1, (1 << 52) + 2, ones - 1, ones - 2]:
        x = Fraction(sig, 1 << 52)
        want = _round(1 / x)
        low = (1 << 105) // sig  # floor of 1/x in units of 2^-53
        one_ulp = Fraction((1 << 15) + 1, 1 << 68)  # and a little
        starts = [k for k in range(low - 2, low + 4)
                  if abs(Fraction(k, 1 << 53) - 1 / x) <= one_ulp]
        assert len(starts) >= 2
        right = []
        for k in starts:
            y = Fraction(k, 1 << 53)
            right.append(_round(y + y * (1 - x * y)) == want)
        assert all(right) or sig == ones, f"significand {sig:#x}"
        if sig == ones:
            assert not all(right)  # the one that pivot_inv selects apart


@pytest.mark.gpu
def test_estimate_and_reciprocals_next_to_midpoints(cuda, tmp_path):
    exe = str(tmp_path / "pivot_estimate_check")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "pivot_estimate_check.cu")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O2", "-std=c++17", "-fmad=false", "-o", exe, src], check=True)
    r = subprocess.run([exe] + [str(x) for x in _significands()], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)
