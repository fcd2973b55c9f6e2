"""The flux's branch-free reciprocal, quotient and root against IEEE float32 (NumPy), bit for bit.

All 2^23 mantissas of the reciprocal and all 2^24 of the root (two binades), at exponents across the stated
range; quotients of random and of awkward operands. The flux itself is compared with the oracle elsewhere.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def probe(a: np.ndarray, b: np.ndarray) -> np.ndarray:
    from inundation_b200 import native

    lib = native.load()
    at, bt = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.empty(3 * a.size, device="cuda")
    native.check(lib.swe_plain_math_probe(at.data_ptr(), bt.data_ptr(), out.data_ptr(), a.size, None), "probe")
    torch.cuda.synchronize()
    return out.cpu().numpy().reshape(3, -1)


def same(x: np.ndarray, y: np.ndarray) -> None:
    bad = np.flatnonzero(x.view(np.uint32) != y.view(np.uint32))
    assert bad.size == 0, (bad.size, x[bad[:4]], y[bad[:4]])


@pytest.mark.parametrize("exponent", [-80, -47, -2, -1, 0, 1, 20, 61])
def test_every_mantissa(exponent: int) -> None:
    mantissas = (np.arange(1 << 23, dtype=np.uint32) | np.uint32((127 + exponent) << 23)).view(np.float32)
    rng = np.random.default_rng(exponent + 100)
    a = (rng.integers(0, 1 << 23, mantissas.size).astype(np.uint32) | np.uint32(127 << 23)).view(np.float32)
    a *= np.where(rng.random(a.size) < 0.5, -1, 1).astype(np.float32)
    got = probe(a, mantissas)
    same(got[0], np.float32(1.0) / mantissas)
    same(got[1], a / mantissas)
    same(got[2], np.sqrt(mantissas))


def test_quotients_of_awkward_operands() -> None:
    rng = np.random.default_rng(3)
    edge = np.array([0, 1, 2, 3, (1 << 23) - 1, (1 << 23) - 2, (1 << 22), (1 << 22) - 1, (1 << 22) + 1], np.uint32)
    m = np.concatenate([edge, rng.integers(0, 1 << 23, 2000).astype(np.uint32)])
    x, y = np.meshgrid(m, m)
    for ea, eb in ((0, 0), (-79, -40), (-79, 40), (60, -40), (60, 20), (5, -47)):
        a = (x.ravel() | np.uint32((127 + ea) << 23)).view(np.float32)
        b = (y.ravel() | np.uint32((127 + eb) << 23)).view(np.float32)
        same(probe(a, b)[1], a / b)
    zero = probe(np.zeros(4, np.float32), np.array([1e-12, 1.0, 3.0, 1e9], np.float32))
    assert (zero[1] == 0.0).all()
    assert (probe(np.ones(1, np.float32), np.zeros(1, np.float32))[2] == 0.0).all()  # the root of zero


@pytest.mark.parametrize("exponent", [-96, -95, -86, -85, -84, -83, -82, -81])
def test_every_mantissa_of_the_root_below_the_quotients_range(exponent: int) -> None:
    """The Roe celerity's argument is g / 2 times a depth of at least 2^-80: 2^-85 for the smallest g that is admitted."""
    mantissas = (np.arange(1 << 23, dtype=np.uint32) | np.uint32((127 + exponent) << 23)).view(np.float32)
    same(probe(np.ones_like(mantissas), mantissas)[2], np.sqrt(mantissas))


@pytest.mark.parametrize("seed", range(4))
def test_quotients_next_to_rounding_boundaries(seed: int) -> None:
    """For mantissas b, the numerators whose quotient lies closest to the middle of two floats on either side: integers
    a with a 2^k = b m + d for odd m (the middle, 25 bits) and odd |d| <= 15, solved for a modulo b's odd part."""
    rng = np.random.default_rng(seed)
    ends = np.concatenate([np.arange(1 << 23, (1 << 23) + 2000), np.arange((1 << 24) - 2000, 1 << 24)])
    b = np.unique(np.concatenate([ends, rng.integers(1 << 23, 1 << 24, 60_000)])).astype(np.int64)
    twos = np.zeros_like(b)
    for _ in range(24):
        twos += (b >> twos) & 1 ^ 1
    odd = b >> twos
    keep = odd > 1
    b, twos, odd = b[keep], twos[keep], odd[keep]
    for k, low, high in ((24, b, np.full_like(b, 1 << 24)), (25, np.full_like(b, 1 << 23), b)):  # a >= b, then a < b
        inverse, base, e = np.ones_like(b), (odd + 1) // 2 % odd, k - twos  # of 2^e modulo the odd part
        for bit in range(5):
            inverse = np.where((e >> bit) & 1, inverse * base % odd, inverse)
            base = base * base % odd
        for d in range(-15, 16, 2):
            a = d % odd * inverse % odd
            a += np.maximum(0, -(-(low - a) // odd)) * odd  # the first of its class in the range
            ok = (a < high) & (e >= 0)
            x, y = a[ok].astype(np.float32), b[ok].astype(np.float32)
            assert x.size > 1000 and (x == a[ok]).all()
            same(probe(x, y)[1], x / y)
