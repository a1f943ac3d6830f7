"""What the int8-slice products (ozaki_i8.cuh) and their guard (slice_guard.cuh)
compute, restated in numpy and checked in exact arithmetic: the byte layout of a
sliced operand, the base-256 digits of the FP64 path, its 34 digit products and
their bounds, and the rule that says which outputs may come from slices.
Changes to either file that alter these statements belong here too."""
from fractions import Fraction

import numpy as np
import pytest

S, W, FIXED, SHIFT, MAXK = 7, 8, 54, 68, 21760       # ozaki::Full
LAYOUTS = [(128, 5), (96, 5), (128, 7), (64, 7)]      # rows per block, slices: A and B of both accuracies


def offset(r, k, s, BR, slices, Kp):
    """Byte of digit s of element (r, k)."""
    chunk = (r // BR * (Kp // 32) + k // 32) * slices * BR * 32
    return chunk + s * BR * 32 + ((r % BR // 8) * 2 + k % 32 // 16) * 128 + r % 8 * 16 + k % 16


@pytest.mark.parametrize("BR,slices", LAYOUTS)
def test_layout(BR, slices):
    Rp, Kp = 3 * BR, 96
    r, k, s = np.meshgrid(np.arange(Rp), np.arange(Kp), np.arange(slices), indexing="ij")
    at = offset(r, k, s, BR, slices, Kp)
    assert np.array_equal(np.sort(at.ravel()), np.arange(Rp * Kp * slices))
    # a chunk of a row block is one contiguous copy, a slab of it 8 x 16 byte core matrices:
    # 128 bytes from one to the next along K, 256 along the rows
    block = at[BR:2 * BR, 32:64, :]
    assert block.max() - block.min() == slices * BR * 32 - 1 and block.min() % (slices * BR * 32) == 0
    slab = at[:BR, :32, 1] - BR * 32
    for i in range(0, BR, 8):
        for j in (0, 16):
            core = slab[i:i + 8, j:j + 16]
            assert np.array_equal(core, i // 8 * 256 + j // 16 * 128 + np.arange(128).reshape(8, 16))


def digits(m):
    """The seven low bytes of (m + c) ^ c, c = 0x80 in each of them; digit 0 the highest."""
    c = 0x0080808080808080
    u = ((int(m) + c) ^ c) & ((1 << 64) - 1)
    d = [(u >> 8 * (6 - s)) & 0xFF for s in range(7)]
    return [x - 256 if x >= 128 else x for x in d]


def test_digits():
    rng = np.random.default_rng(1)
    edge = [0, 1, -1, 127, 128, 129, -127, -128, -129, 1 << 53, -(1 << 53), 1 << 54, -(1 << 54), (1 << 54) - 1,
            0x7F7F7F7F7F7F7F, -0x7F7F7F7F7F7F7F, 0x00808080808080, -0x00808080808080]
    edge = [m for m in edge if abs(m) <= 1 << 54]
    for m in edge + [int(x) for x in rng.integers(-(1 << 54), (1 << 54) + 1, 3000)]:
        d = digits(m)
        assert sum(x * 256 ** (6 - s) for s, x in enumerate(d)) == m
        assert abs(d[0]) <= 65 and all(-128 <= x <= 127 for x in d)
        assert abs(m / 2.0 ** 48 - d[0]) <= 0.503        # the leading digit: what the guard's means are made of


def test_accumulators_fit_32_bits():
    # accumulator w holds the pairs s + t = w; digit 0 is at most 65, the others 128
    for w in range(W):
        worst = sum((65 if s == 0 else 128) * (65 if w - s == 0 else 128) for s in range(S) if 0 <= w - s < S)
        assert worst * MAXK < 1 << 31
    assert sum(1 for s in range(S) for t in range(S) if s + t < W) == 34
    # what the dropped pairs can add to a term of 2^{e_x + e_y}
    assert sum(2.0 ** 14 * 2.0 ** (8 * (7 - s - t) - SHIFT) for s in range(S) for t in range(S) if s + t >= W) < 2.0 ** -59


def exponents(X):
    return np.frexp(np.abs(X).max(axis=1))[1]


def sliced(X, Y):
    """The sliced product: exact sums of the 34 digit products, one rounding."""
    ex, ey = exponents(X), exponents(Y)
    cut = lambda A, e: np.array([[digits(np.rint(np.ldexp(a, FIXED - e[r]))) for a in A[r]] for r in range(len(A))])
    dx, dy = cut(X, ex), cut(Y, ey)
    out = np.zeros((len(X), len(Y)))
    for i in range(len(X)):
        for j in range(len(Y)):
            T = sum(int(dx[i, :, s] @ dy[j, :, t]) << 8 * (7 - s - t) for s in range(S) for t in range(S) if s + t < W)
            out[i, j] = float(Fraction(T) * Fraction(2) ** int(ex[i] + ey[j] - SHIFT))
    return out


def chain(X, Y):
    """FP64 multiply-adds along k (80-bit products, rounded to FP64 per step)."""
    acc = np.zeros((len(X), len(Y)))
    for k in range(X.shape[1]):
        acc = np.float64(acc + X[:, k].astype(np.longdouble)[:, None] * Y[:, k].astype(np.longdouble)[None, :])
    return acc


def taken(X, Y):
    """The guard's rule per output."""
    ex, ey = exponents(X), exponents(Y)
    q = lambda A, e: np.ldexp(np.abs(A), -e[:, None]) ** 2
    mean = lambda A, e: (np.mean(np.rint(np.ldexp(A, 6 - e[:, None])) ** 2, axis=1) + 0.25) / 4096.0
    return q(X, ex) @ q(Y, ey).T >= 0.25 * (mean(X, ex)[:, None] + mean(Y, ey)[None, :])


def errors(X, Y):
    ref = [[sum(Fraction(float(a)) * Fraction(float(b)) for a, b in zip(x, y)) for y in Y] for x in X]
    off = lambda R: np.array([[float(abs(Fraction(float(R[i, j])) - ref[i][j])) for j in range(len(Y))]
                              for i in range(len(X))])
    return off(sliced(X, Y)), off(chain(X, Y))


def rows(kind, K, rng, n=10):
    X, Y = rng.standard_normal((n, K)), rng.standard_normal((n, K))
    even = np.arange(K) % 2 == 0
    if kind == "graded":
        w = 10.0 ** (-6.0 * np.arange(K) / K)
        return X * w, Y * w
    if kind == "same sign":
        return np.abs(X), np.abs(Y)
    if kind == "heavy tails":
        return X ** 5, Y
    if kind.startswith("apart"):
        c = float(kind.split()[1])
        return X * np.where(even, 1.0, c), Y * np.where(even, c, 1.0)
    return X, Y


@pytest.mark.parametrize("K", [60, 240])
@pytest.mark.parametrize("kind", ["gauss", "graded", "same sign", "heavy tails", "apart 0.3", "apart 1e-1", "apart 1e-2",
                                  "apart 1e-6"])
def test_guard_keeps_what_is_better(kind, K):
    """rms error of the outputs taken from slices: at most the chain's.  (The rule
    is set where the two are equal for independent roundings; 100 outputs.)"""
    X, Y = rows(kind, K, np.random.default_rng(K))
    ok = taken(X, Y)
    if kind in ("gauss", "same sign"):
        assert ok.all()
    if kind in ("apart 1e-2", "apart 1e-6"):
        assert not ok.any()
    es, ec = errors(X, Y)
    if ok.any():
        assert np.sqrt(np.mean(es[ok] ** 2)) <= np.sqrt(np.mean(ec[ok] ** 2))
    if kind == "apart 1e-6":
        assert np.sqrt(np.mean(es ** 2)) > 1e3 * np.sqrt(np.mean(ec ** 2))   # what the guard is for
