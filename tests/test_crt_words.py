"""The CRT's arithmetic up to its 64-bit words (csrc/crt.cuh, crt_limbs),
modelled on the CPU for every modulus count: t stored as BF16, limb sums and
quotient in FP32, limbs converted to integers and four of them gathered in a
word. (crt_limb_model.py keeps the earlier form: t stored with a bias, carries
between FP32 digits; its tables, FP32 steps and the epilogue's reduction are
the kernel's still.)
"""
import numpy as np
import pytest

import crt_limb_model as CL
from test_crt_round import words


def kernel_words(T, r):
    """The three words of the value with residues r, every exact step checked."""
    S = [np.float32(0)] * T.NP
    for i, m in enumerate(T.m):
        t = np.float32(CL.gemm_t(r[i] * T.inv[i], m))  # the GEMM's sum is congruent to r inv
        stored = int(t.view(np.uint32)) >> 16          # the upper half of the float: BF16
        assert np.uint32(stored << 16).view(np.float32) == t and abs(t) <= 182
        for j in range(T.NP):
            exact = int(S[j]) + int(t) * T.Pd[i][j]
            S[j] = CL.fma32(t, np.float32(T.Pd[i][j]), S[j])
            assert int(S[j]) == exact and abs(exact) < 2**23.5
    est = np.float32(0)
    for j in sorted(T.c, reverse=True):
        est = CL.fma32(S[j], T.c[j], est)
    q = (est + CL.MAGIC) - CL.MAGIC
    Y = [0] * 12
    for j in range(T.NP + 1):
        exact = (int(S[j]) if j < T.NP else 0) - int(q) * T.Md[j]
        assert float(CL.fma32(q, np.float32(-T.Md[j]), S[j] if j < T.NP else np.float32(0))) == exact
        assert abs(exact) < 2**23.5
        Y[j] = exact
    return words(Y)


@pytest.mark.parametrize("q", list(range(8, 16)))
def test_words_are_the_value(q):
    T = CL.Table(q)
    rng = np.random.default_rng(700 + q)
    bound = T.M * 15 // 32
    values = [0, 1, -1, bound, -bound, T.M // 3, -(T.M // 4)]
    values += [int.from_bytes(rng.bytes(16), "little") % (2 * bound) - bound for _ in range(200)]
    residues = [[y % m for m in T.m] for y in values]
    # every t near its largest, as far as the value stays inside the margin
    residues += [[int(rng.choice([0, m // 2, (m + 1) // 2, m - 1, 1])) for m in T.m] for _ in range(400)]
    tried = 0
    for r in residues:
        y = CL.symmetric_crt(T, r)
        if abs(y) <= bound:
            tried += 1
            w = kernel_words(T, r)
            assert sum(v << (52 * g) for g, v in enumerate(w)) == y
    assert tried > 250
