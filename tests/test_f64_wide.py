"""Bounds of the wide FP64 rows (primes below 1.1 2^50; fhb_pass.cuh): each
pass of four butterfly stages, on the worst operands its inputs allow, keeps
every value exact (below 2^53) and every quotient below the rounding
constant's reach (2^51), and leaves words that its reductions bring back to
what the next pass assumes.  Exact integers; only the quotient is rounded in
double precision, as on the device."""

from fractions import Fraction

import numpy as np
import pytest

from fhelium_b200.config import CkksConfig, Preset

LIMIT = 11 * (1 << 50) // 10
ROUND = 6755399441055744.0  # 1.5 2^52


def _primes():
    qs = [int(q) for q in CkksConfig.parse(Preset.slots32768_scale50_levels27_int64).q_moduli if int(q) < LIMIT]
    assert len(qs) >= 27
    return qs[::6] + [LIMIT - 1]  # and the largest modulus the form admits


def _rounded(x: int, y: float) -> int:
    """fma(x, y, ROUND) - ROUND for a double x (an integer) and a double y."""
    exact = Fraction(float(x)) * Fraction(y)
    assert abs(exact) < 1 << 51
    return round(exact)


def _product(x: int, w: int, q: int) -> int:
    h = float(x * w)  # correctly rounded
    r = x * w - _rounded(int(h), 1.0 / q) * q
    assert abs(r) < 1 << 53
    return r


def _by_constant(x: int, w: int, q: int) -> int:
    """A product by a constant kept with w / q (0 <= w < q)."""
    r = x * w - _rounded(x, w / q) * q
    assert abs(r) < 1 << 53
    return r


def _reduce(x: int, q: int) -> int:
    assert abs(x) < 1 << 53
    r = x - _rounded(x, 1.0 / q) * q
    assert abs(r) <= 0.51 * q
    return r


def _worst(bound: float, q: int, rng) -> list[int]:
    b = int(bound * q)
    return [b, -b, b - 1, q // 2, -(q // 2), 0] + [int(v) for v in rng.integers(-b, b, 10)]


def _twiddles(q: int, rng) -> list[int]:
    half = q // 2
    return [half, -half, half - 1, 1, -1] + [int(v) for v in rng.integers(-half, half, 6)]


@pytest.mark.parametrize("start,stated", [(1.0, (1.64, 2.37, 3.19, 4.13)), (0.51, (1.09, 1.74, 2.48, 3.33))])
def test_forward_pass_of_four_stages(start, stated):
    """`stated`: the bounds after each stage, over q, of the largest modulus."""
    rng = np.random.default_rng(3)
    for q in _primes():
        bound = start
        for after in stated:
            assert bound + 0.5 + bound * 1.1 / 8 <= after
            xs, top = _worst(bound, q, rng), 0
            for y in xs:
                for w in _twiddles(q, rng):
                    top = max(top, abs(_product(y, w, q)))
            assert top <= (0.5 + bound * 1.1 / 8 + 1e-3) * q
            bound = min(after, bound + 0.5 + bound * 1.1 / 8)
            assert bound * q < 1 << 53
        for x in _worst(bound, q, rng):
            _reduce(x, q)


def test_inverse_pass_of_four_stages():
    rng = np.random.default_rng(4)
    for q in _primes():
        grown = [0.51] * 16  # bound of each word over q
        for stage in range(4):
            nxt = list(grown)
            for i in range(16):
                j = i | (1 << stage)
                if i == j:
                    continue
                total = grown[i] + grown[j]
                assert total * q < 1 << 53
                top = max(abs(_product(d, w, q)) for d in _worst(total, q, rng)[:6] for w in _twiddles(q, rng)[:5])
                nxt[i], nxt[j] = total, max(top / q, 0.5 + total * 1.1 / 8)
            grown = nxt
            assert max(grown) <= (1.02, 2.04, 1.57, 3.13)[stage]
            if stage == 1:
                grown = [0.51 if (i & 3) < 2 else g for i, g in enumerate(grown)]
        for g in grown:
            for x in _worst(g, q, rng):
                _reduce(x, q)


def test_key_products_and_their_sums():
    """Key words enter as u - q.  The rows launch multiplies reduced words, or
    own-digit words (a product by R^-1 of a word u - q, 0.64 q at most): four
    terms of 0.68 q on a reduced sum.  The application of hoisted rotations
    multiplies words u - q themselves: four terms of 0.78 q."""
    rng = np.random.default_rng(5)
    for q in _primes():
        keys = [q - 1, -q, 1 - q, q // 3]
        own = max(abs(_by_constant(x, w, q)) for x in _worst(1.0, q, rng)
                  for w in [q - 1, q - 2, q // 2, 1] + [int(v) for v in rng.integers(0, q, 12)])
        assert own <= 0.64 * q
        for start, term in ((0.64, 0.68), (1.0, 0.78)):
            top = max(abs(_product(x, k, q)) for x in _worst(start, q, rng) for k in keys)
            assert top <= (0.5 + start * 1.1 / 4 + 1e-3) * q <= term * q
            assert (0.51 + 4 * term) * q < 1 << 53
