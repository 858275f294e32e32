"""The arithmetic of the integer pair products (k_crt.cu) on the host: moduli, residues through FP32
dot products of 16-bit limbs, the bytes of the INT32 accumulators and the way back, with the constants
the kernels use, in the same operations."""
import math
import os
import re

import numpy as np

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gaspacho2_b200", "csrc", "k_crt.cu")
TEXT = open(SRC).read()
MODULI = [int(v) for v in re.search(r"kModuli\[kMod\] = \{([^}]*)\}", TEXT).group(1).split(",")]
MAX_K = int(re.search(r"kMaxK = (\d+)", TEXT).group(1))
PRODUCT = math.prod(MODULI)
R = math.sqrt(0.48 * PRODUCT)


def _centred(v, p):
    v %= p
    return v - p if 2 * v > p else v


def _residues(x, p, y):
    """crt_limbs and crt_residue for an array of integers (Python ints) x: the low bytes as INT8."""
    limbs = []
    for _ in range(3):
        low = [((v + 32768) & 0xFFFF) - 32768 for v in x]
        limbs.append(low)
        x = [(v - b) >> 16 for v, b in zip(x, low)]
    limbs.append(x)
    f = np.float32
    acc = None
    for q in (3, 2, 1, 0):  # every partial sum is an integer below 2^24: exact in FP32
        c = _centred(pow(2, 16 * q, p) * y, p)
        term = [a * c for a in limbs[q]]
        acc = term if acc is None else [s + t for s, t in zip(acc, term)]
        assert max(abs(v) for v in acc) < 2 ** 24
    v = np.array(acc, f)
    rnd = f(12582912.0)
    t = (v.astype(np.float64) * np.float64(f(1.0) / f(p)) + np.float64(rnd)).astype(f)  # one rounding, as fmaf
    r = (v.astype(np.float64) - np.float64(p) * (t - rnd).astype(np.float64)).astype(np.int64)
    assert p == 256 or np.abs(r).max() <= 127
    return ((r + 128) & 255) - 128


def test_moduli():
    assert MODULI[0] == 256 and all(p <= 253 for p in MODULI[1:])
    assert all(math.gcd(a, b) == 1 for i, a in enumerate(MODULI) for b in MODULI[:i])
    assert R < 2.0 ** 60  # the scaled integers fit the four limbs
    assert MAX_K * 2 ** 14 < 2 ** 31 - 256 and MAX_K % 256 == 0


def test_products_of_integers():
    rng = np.random.default_rng(1)
    K = 300
    for scale in (1.0, 1e-3, 1e-9):  # rows at the norm limit and far below it
        a, b = rng.standard_normal(K), rng.standard_normal(K) + 0.3
        a, b = a / np.linalg.norm(a), b / np.linalg.norm(b)
        x = [int(v) for v in np.rint(a * R * scale)]
        w = [int(v) for v in np.rint(b * R * 0.999)]
        exact = sum(p * q for p, q in zip(x, w))
        s = 0
        for p in MODULI:
            y = pow(PRODUCT // p, -1, p)
            acc = int(np.sum(_residues(x, p, y) * _residues(w, p, 1)))  # INT32 in the tensor core
            off, magic = (2 ** 31 + p - 1) // p * p, 2 ** 39 // p
            u = acc + off
            byte = u - ((u * magic) >> 39) * p
            assert 0 <= byte < 256 and (byte - acc * 1) % p == 0
            f = ((1 << 80) + p // 2) // p
            s += byte * f
        frac = ((s + 2 ** 15) >> 16) % 2 ** 64
        frac -= 2 ** 64 if frac >= 2 ** 63 else 0
        got = frac * (PRODUCT / 2.0 ** 64)
        assert abs(got - exact) <= 2.0 ** -52 * abs(exact) + PRODUCT * 2.0 ** -63


def test_accumulator_bytes_over_the_whole_range():
    rng = np.random.default_rng(2)
    edge = MAX_K * 2 ** 14
    x = np.concatenate([rng.integers(-edge, edge + 1, 200000), [-edge, edge, 0, -1, 1]])
    for p in MODULI:
        off, magic = (2 ** 31 + p - 1) // p * p, 2 ** 39 // p
        u = (x + off).astype(np.uint64)
        assert u.max() < 2 ** 32
        r = u - ((u * np.uint64(magic)) >> np.uint64(39)) * np.uint64(p)
        assert r.max() < 256 and np.all((r.astype(np.int64) - x) % p == 0)


def test_extreme_limbs():
    big = int(R)
    x = [big, -big, 2 ** 47, -(2 ** 47), 2 ** 31, 2 ** 15, -(2 ** 15), 32767, 0, 1, -1, big // 2, (1 << 53) - 1]
    for p in MODULI:
        for y in (1, pow(PRODUCT // p, -1, p)):
            r = _residues(x, p, y)
            assert all((int(a) - b * y) % p == 0 for a, b in zip(r, x))
