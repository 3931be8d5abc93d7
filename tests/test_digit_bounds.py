"""Why the tensor-core kernel may combine its four int32 levels in pairs
(quad_sum, tc_mixed.cu): over all digit words of |X| <= 2^30 a product of two
words adds at most 8371968 to 2^8 L2 + L3 and 2^20 to 2^8 L0 + L1, so that
sums of 256 products stay below 2^31.  Each level is linear in every digit, so
the ends of the digits' ranges decide, which are enumerated here."""
import itertools

import numpy as np

K = 256  # products of one accumulation run: a batch's points


def digits(X):
    """the four balanced base-256 digits of X, leading one first (digits_word, tc_ptx.cuh)"""
    out = []
    for _ in range(3):
        d = (X + 128) % 256 - 128
        out.append(d)
        X = (X - d) // 256
    return (X, *out[::-1])


def value(d):
    return ((d[0] * 256 + d[1]) * 256 + d[2]) * 256 + d[3]


def ends():
    """ends of the ranges of the digits: |d0| <= 63 with the others free, and
    |d0| = 64 with the rest on the other side of zero"""
    free = (-128, 127)
    words = [(d0, *r) for d0 in (-63, 63) for r in itertools.product(free, repeat=3)]
    words += [(64, d1, *r) for d1 in (-128, -1) for r in itertools.product(free, repeat=2)]
    words += [(64, 0, d2, d3) for d2 in (-128, -1) for d3 in free] + [(64, 0, 0, d3) for d3 in (-128, 0)]
    words += [(-64, d1, *r) for d1 in (1, 127) for r in itertools.product(free, repeat=2)]
    words += [(-64, 0, d2, d3) for d2 in (1, 127) for d3 in free] + [(-64, 0, 0, d3) for d3 in (0, 127)]
    return words


def test_pairs_of_levels_fit_int32():
    W = ends()
    assert all(abs(value(w)) <= 2 ** 30 and digits(value(w)) == w for w in W)
    d, e = np.array(W)[:, None, :], np.array(W)[None, :, :]
    level = [sum(d[..., i] * e[..., L - i] for i in range(L + 1)) for L in range(4)]
    a, b = 256 * level[0] + level[1], 256 * level[2] + level[3]
    assert abs(a).max() == 2 ** 20 and abs(b).max() == 8371968
    for s in (a, b, 256 * level[0], 256 * level[2]):
        assert K * abs(s).max() < 2 ** 31


def test_every_word_is_within_the_ends():
    rng = np.random.default_rng(0)
    for X in [int(x) for x in rng.integers(-2 ** 30, 2 ** 30 + 1, 20000)] + [2 ** 30, -2 ** 30, 2 ** 30 - 2 ** 23]:
        w = digits(X)
        assert value(w) == X and abs(w[0]) <= 64 and all(-128 <= d <= 127 for d in w[1:])
        assert abs(w[0]) < 64 or w[0] * value((0, *w[1:])) <= 0
