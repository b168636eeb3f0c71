"""CPU checks of the exact-accumulation scheme's restatement (oracle/ozaki_oracle.py):
the slicing is exact, the level sums stay on their grids, and the result is
the FP64 product up to the final rounding."""
import numpy as np
import pytest

from oracle import ozaki_oracle as Z


def rand(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def test_pairs_are_levels_up_to_four():
    assert len(Z.PAIRS) == 15
    assert all(i + j <= 4 for i, j in Z.PAIRS)
    assert len(set(Z.PAIRS)) == 15


def test_slices_exact_in_bf16_and_reconstruct():
    rng = np.random.default_rng(0)
    x = rng.uniform(-1, 1, 100000)
    x[:5] = [0.0, -0.999999940395, 0.999999940395, 2.0 ** -40, -(2.0 ** -8)]
    s = Z.slices(x)
    for i, si in enumerate(s):
        assert Z.bf16_exact(si)
        g = 2.0 ** (7 * (i + 1))
        assert np.all(np.rint(si * g) == si * g)  # on the slice grid
        assert np.all(np.abs(si) <= (1.0 if i == 0 else 2.0 ** (-7 * i - 1)))
    assert np.max(np.abs(x - sum(s))) <= 2.0 ** -36


def test_row_exponents_bound_rows():
    rng = np.random.default_rng(1)
    X = rand(rng, (50, 40)) * np.exp2(rng.integers(-50, 50, size=(50, 1)))
    X[3] = 0
    e = Z.row_exponents(X)
    assert e[3] == Z.ZERO_EXP
    live = e != Z.ZERO_EXP
    m = np.maximum(np.abs(X.real), np.abs(X.imag)).max(axis=1)
    assert np.all(m[live] < np.exp2(e[live].astype(float)))
    assert np.all(m[live] >= np.exp2(e[live].astype(float) - 1))


def test_level_sums_on_exact_grids_for_k512():
    rng = np.random.default_rng(2)
    A = rand(rng, (16, 512))
    B = rand(rng, (512, 8))
    _, lv = Z.ozaki_matmul(A, B)
    for part in (lv[0].real, lv[0].imag):
        assert np.all(np.rint(part * 2.0 ** 14) == part * 2.0 ** 14)
        assert np.max(np.abs(part)) * 2.0 ** 14 < 2.0 ** 24  # fits the FP32 significand
    for part in (lv[1].real, lv[1].imag):
        assert np.all(np.rint(part * 2.0 ** 21) == part * 2.0 ** 21)
        assert np.max(np.abs(part)) * 2.0 ** 21 < 2.0 ** 24


def test_result_is_rounded_fp64_product():
    rng = np.random.default_rng(3)
    A = rand(rng, (64, 256)).astype(np.complex64).astype(np.complex128)
    B = rand(rng, (256, 48))
    C, _ = Z.ozaki_matmul(A, B)
    ref = A @ B
    assert np.all(np.abs(C - ref) <= Z.error_bound(A, B, ref))


# ---- four fp16 slices ----------------------------------------------------------

def cancelling(rng, m, k, n):
    """Rows and columns whose leading slices cancel over K while the next ones
    do not: level 0 is small, level 1 is large."""
    a = np.where(np.arange(k) % 2 == 0, 0.75, -0.75) + 0.95 * 2.0 ** -8
    A = np.tile(a, (m, 1)) * (1 + 0j)
    A[m // 2:] *= 1j
    b = np.repeat(rng.uniform(0.9, 1.0, (k // 2, n)), 2, axis=0)
    return (A.astype(np.complex64).astype(np.complex128), b.astype(np.complex64).astype(np.complex128))


@pytest.mark.parametrize("k", [16, 128, 129, 256])
@pytest.mark.parametrize("side", [0, 1])
def test_half_slices_are_fp16_and_reconstruct(k, side):
    """Each slice is an fp16 value (times 2^15), slices 0 and 1 lie on their
    grids, every slice is at most half a step of the one before, and the
    residual is at most 2^-39 (2^-36 for five bf16 slices)."""
    rng = np.random.default_rng(k + side)
    x = rng.uniform(-1, 1, 200000) * np.exp2(-rng.integers(0, 20, 200000))
    x[:4] = [0.0, 1 - 2.0 ** -53, -(1 - 2.0 ** -24), 2.0 ** -39]
    b0, more = Z.half_bits(k, side)
    s = Z.half_slices(x, k, side)
    for v in s[:3]:
        assert np.all(np.float64(np.float16(v * 2.0 ** 15)) == v * 2.0 ** 15)
    for v, g in zip(s[:2], (b0, b0 + more)):
        assert np.all(np.rint(v * 2.0 ** g) == v * 2.0 ** g)
    assert np.max(np.abs(s[1])) <= 2.0 ** -(b0 + 1) and np.max(np.abs(s[2])) <= 2.0 ** -(b0 + more + 1)
    assert np.max(np.abs(x - sum(s))) <= 2.0 ** -39


@pytest.mark.parametrize("k", [16, 100, 128, 129, 200, 256])
def test_half_level_sums_fit_the_significand(k):
    """The largest sums that levels 0 and 1 can reach (every slice at its
    largest, all signs alike) are at most 2^24 steps of their grids."""
    (a0, am), (b0, bm) = Z.half_bits(k, 0), Z.half_bits(k, 1)
    assert 2 * k <= 2.0 ** (24 - a0 - b0)
    grid = max(a0 + b0 + bm, a0 + am + b0)
    assert 2 * k * (2.0 ** -(a0 + 1) + 2.0 ** -(b0 + 1)) <= 2.0 ** (24 - grid)


@pytest.mark.parametrize("k", [16, 64, 128, 144, 256])
@pytest.mark.parametrize("kind", ["random", "binades", "cancelling", "equal"])
def test_half_split_is_no_less_exact_than_five_slices(k, kind):
    """The tensor core's sums of either split against the product in extended
    precision: the fp16 split's rms error is no larger, and each element is within
    error_bound."""
    rng = np.random.default_rng(k)
    m, n = 48, 40
    A, B = rand(rng, (m, k)), rand(rng, (k, n))
    if kind == "binades":
        A = A * np.exp2(-rng.integers(0, 21, (m, k)))
        B = B * np.exp2(-rng.integers(0, 21, (k, n)))
    elif kind == "cancelling":
        A, B = cancelling(rng, m, k, n)
    elif kind == "equal":
        A, B = np.full((m, k), (1 + 1j) * (1 - 2.0 ** -13)), np.full((k, n), (1 + 1j) * (1 - 2.0 ** -12))
    ref = (A.astype(np.clongdouble) @ B.astype(np.clongdouble)).astype(np.complex128)
    e4 = np.abs(Z.accumulate(A, B, True) - ref)
    e5 = np.abs(Z.accumulate(A, B, False) - ref)
    assert np.sqrt(np.mean(e4 ** 2)) <= np.sqrt(np.mean(e5 ** 2))
    assert np.all(e4 <= Z.error_bound(A, B, ref))


def test_half_pairs_and_dropped_terms():
    """The pairs that the fp16 split leaves out are, with the residuals, at most
    what five slices leave out: 2^-34 of the scales per product."""
    for k in (16, 128, 129, 256):
        size = []
        for side in (0, 1):
            b0, more = Z.half_bits(k, side)
            s2 = b0 + more + 1
            size.append([0, b0 + 1, s2, s2 + 12])
        out = sum(2.0 ** -(size[0][i] + size[1][j]) for i in range(4) for j in range(4) if (i, j) not in Z.HALF_PAIRS)
        assert out + 2 * 2.0 ** -39 < 2.0 ** -34


def test_five_slices_bound_cancelling_rows():
    rng = np.random.default_rng(4)
    A, B = cancelling(rng, 8, 512, 8)
    ref = A @ B
    assert np.all(np.abs(Z.accumulate(A, B, False) - ref) <= Z.error_bound(A, B, ref))
