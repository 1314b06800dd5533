"""The CRT's rounding on FP64 additions (csrc/crt.cuh, crt_round_add), modelled
in Python integers and doubles: for up to 13 moduli the reconstructed integer,
given as limbs of weight 2^(13 j), must come out as its one correct rounding
(Python's int -> float), and every intermediate must stay in its stated range.
"""
import struct

import numpy as np
import pytest

import crt_limb_model as CL


def bits(b):
    return struct.unpack("<d", struct.pack("<Q", b & (2**64 - 1)))[0]


def s64(v):
    return (v + 2**63) % 2**64 - 2**63


def words(limbs):
    """Four limbs to a word, as the kernel's 64-bit multiply-adds leave them."""
    out = []
    for g in range(3):
        v = sum(y << (13 * j) for j, y in enumerate(limbs[4 * g:4 * g + 4]))
        assert abs(v) < 2**63
        out.append(v)
    return out


def rounded(limbs):
    w0, w1, w2 = words(limbs)
    V = s64(w1 + (w0 >> 52) + (w2 << 52))
    low = w0 % 2**52
    assert sum(y << (13 * j) for j, y in enumerate(limbs)) == (V << 52) + low
    if -(2**32) <= V < 2**32:
        a = bits(low | 0x433 << 52) - 2.0**52
        assert a == low
        return float((V << 52) + int(a))  # one fused multiply-add of exact operands
    a52 = (low >> 6) | ((V & 63) << 46) | (1 if low & 63 else 0)
    B = V >> 6
    assert abs(B) < 2**51
    x = bits(((1023 + 52 + 58) << 52 | 1 << 51) + B) - (1.5 * 2.0**52 + 1.0) * 2.0**58
    assert int(x) == (B - 1) << 58
    return x + bits((1023 + 58) << 52 | a52)


def limbs_of(y, np_, rng, spread):
    """Limbs of y with random carries left in them (|limb| < 2^23.5)."""
    d = [0] * 12
    rest = y
    for j in range(np_):
        r = (rest + 4096) % 8192 - 4096
        rest = (rest - r) >> 13
        d[j] = r
    d[np_] = rest
    for j in range(np_):
        c = int(rng.integers(-spread, spread + 1))
        d[j] += c << 13
        d[j + 1] -= c
    assert sum(v << (13 * j) for j, v in enumerate(d)) == y and max(abs(v) for v in d) < 2**23.5
    return d


@pytest.mark.parametrize("q", [8, 9, 11, 12, 13])
def test_one_correct_rounding(q):
    T = CL.Table(q)
    bound = T.M * 15 // 32
    rng = np.random.default_rng(q)
    values = [0, 1, -1, bound, -bound]
    for p in (51, 52, 53, 57, 58, 59, 60, 61, 83, 84, 85, 90, 100, 107, 108):
        for m in (2**52 + 1, 2**53 - 1, 2**52, int(rng.integers(2**52, 2**53))):
            top = m << p >> 52  # around 2^p, 53 significant bits
            for d in (0, 1, -1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 1 << max(p - 53, 0), (1 << max(p - 53, 0)) + 1,
                      (1 << max(p - 53, 0)) - 1, 3 << max(p - 53, 0)):
                values += [top + d, -(top + d)]
    for _ in range(20000):
        v = int.from_bytes(rng.bytes(14), "little") % (2 * bound) - bound
        values.append(v >> int(rng.integers(0, T.M.bit_length())))
    for y in values:
        if abs(y) <= bound:
            assert rounded(limbs_of(y, T.NP, rng, 1100)) == float(y), y
