"""The CRT's rounding for every modulus count (csrc/crt.cuh, crt_round_add), modelled
in Python integers and doubles: the reconstructed integer, given as limbs of
weight 2^(13 j), is cut into an upper and a lower half, each becomes a double
through its bits, and their sum must be its one correct rounding (Python's int
-> float). Values sit around the line between the two forms, the ranges' ends
and the halves of an ulp.
"""
import numpy as np
import pytest

import crt_limb_model as CL
from test_crt_round import bits, limbs_of, s64, words


def rounded(q, limbs):
    sh = 0 if q <= 12 else {13: 6, 14: 14, 15: 23}[q]
    fold = (1 << sh) - 1
    w0, w1, w2 = words(limbs)
    low, mid = w0 % 2**52, w1 + (w0 >> 52)
    assert abs(mid) < 2**63
    B = s64((mid >> sh) + (w2 << 52 - sh))
    assert abs(B) < 2**51
    if q <= 12 or -(1 << 32 - sh) <= B < 1 << 32 - sh:
        V = B << sh | mid & fold
        assert sum(y << (13 * j) for j, y in enumerate(limbs)) == (V << 52) + low
        upper = bits(((1023 + 104) << 52 | 1 << 51) + V) - (1.5 * 2.0**104 + 2.0**52)
        lower = bits(low | (1023 + 52) << 52)
        assert int(upper) == (V - 1) << 52 and int(lower) == 2**52 + low
    else:
        rest = (mid & fold) << 52 | low
        assert sum(y << (13 * j) for j, y in enumerate(limbs)) == (B << 52 + sh) + rest
        cut = (mid & fold) << 52 - sh | low >> sh | (1 if low & fold else 0)
        assert cut | 1 == rest >> sh | 1 and cut < 2**52
        upper = bits(((1023 + 104 + sh) << 52 | 1 << 51) + B) - (1.5 * 2.0**52 + 1.0) * 2.0**(52 + sh)
        lower = bits(cut | (1023 + 52 + sh) << 52)
        assert int(upper) == (B - 1) << 52 + sh
    return upper + lower


@pytest.mark.parametrize("q", list(range(8, 16)))
def test_one_correct_rounding(q):
    T = CL.Table(q)
    bound = T.M * 15 // 32
    rng = np.random.default_rng(q)
    values = [0, 1, bound, bound - 1, 2**52, 2**52 - 1]
    for p in range(51, T.M.bit_length()):
        for m in (2**52, 2**52 + 1, 2**53 - 1, int(rng.integers(2**52, 2**53))):
            top = m << p >> 52  # around 2^p, 53 significant bits
            half = 1 << max(p - 53, 0)
            values += [top + d for d in (0, 1, -1, half, half + 1, half - 1, 3 * half, 3 * half - 1)]
    for _ in range(4000):
        v = int.from_bytes(rng.bytes(16), "little") % bound
        values.append(v >> int(rng.integers(0, bound.bit_length())))
    for y in values:
        if y <= bound:
            assert rounded(q, limbs_of(y, T.NP, rng, 1100)) == float(y), y
            assert rounded(q, limbs_of(-y, T.NP, rng, 1100)) == -float(y), y
