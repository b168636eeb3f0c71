"""FP64 CPU restatement of the exact-accumulation tensor-core contraction
(PQ_PREC_OZAKI) -- test infrastructure only.

The Ozaki scheme (Ozaki, Ogita, Oishi, Rump, "Error-free transformations of
matrix multiplication by using fast routines of matrix multiplication and its
applicability", Numer. Algorithms 59, 2012) as the library runs it:

* every row of A (over K) and every column of B is scaled by 2^-e, e the
  frexp exponent of the largest |Re| or |Im| of that row / column;
* a scaled value x in (-1, 1) is cut into five slices
  s0 = rint(x 2^7) 2^-7, s_i = rint((x - s0 - ... - s_{i-1}) 2^{7(i+1)}) 2^{-7(i+1)};
* the complex product is formed from the 15 slice pairs (i, j) with
  i + j <= 4, summed per level 0, 1 and 2-4; level 0 and 1 sums are exact
  (FP32 on the device, FP64 here), and the result is
  (L0 + L1 + L2) 2^(ea + eb) rounded once to the output type.

Level-0 and level-1 sums are exact in both places, so the device result
equals ``ozaki_matmul`` up to the FP32 rounding of the small level-2-4 sum
(about 2^-30 relative) before the final rounding.

For complex64 results with K <= 256 the device cuts four fp16 slices instead
(``half_slices``): s0 and s1 on fixed grids chosen so that levels 0 and 1 are
exact again, s2 the remainder rounded to fp16's 11 bits and s3 the rest of
that; 11 slice pairs (``HALF_PAIRS``).  Its residual and the pairs it drops are
smaller than the five-slice scheme's, so ``error_bound`` holds for both.
``accumulate`` restates the tensor core's sums of either split in the
kernel's order (additions truncated to FP32's 24 bits).
"""
from __future__ import annotations

import numpy as np

N_SLICES = 5
BITS = 7


def pairs(n_slices=N_SLICES):
    """Slice pairs (i, j) with i + j < n_slices (15 for five slices, 6 for
    the three of PQ_PREC_3XBF16)."""
    return [(i, lvl - i) for lvl in range(n_slices) for i in range(lvl + 1)]


PAIRS = pairs()
ZERO_EXP = -4096


def row_exponents(X):
    """frexp exponent of max(|Re|, |Im|) over each row of X (rows x K);
    ZERO_EXP for an all-zero row."""
    m = np.maximum(np.abs(X.real), np.abs(X.imag)).max(axis=1)
    e = np.frexp(m)[1].astype(np.int64)
    e[m == 0] = ZERO_EXP
    return e


def slices(x, n_slices=N_SLICES):
    """The fixed-grid slices of x (|x| < 1), each exact in bf16."""
    out = []
    r = np.array(x, dtype=np.float64)
    for i in range(n_slices):
        g = 2.0 ** (BITS * (i + 1))
        s = np.rint(r * g) / g
        out.append(s)
        r = r - s
    return out


def bf16_exact(v):
    """True where v is exactly representable in bf16 (8 significant bits)."""
    v = np.asarray(v, dtype=np.float64)
    m, _ = np.frexp(v)
    return np.all(np.rint(m * 256) == m * 256)


def ozaki_matmul(A, B, out_dtype=np.complex64, n_slices=N_SLICES):
    """C = A @ B (A: M x K, B: K x N complex) the way the device computes it;
    returns (C rounded to out_dtype, levels (L0, L1, L2) complex, unscaled)."""
    ea = row_exponents(A)
    eb = row_exponents(B.T)
    sa = np.where(ea == ZERO_EXP, 0, -ea).astype(np.float64)
    sb = np.where(eb == ZERO_EXP, 0, -eb).astype(np.float64)
    As = A * np.exp2(sa)[:, None]
    Bs = B * np.exp2(sb)[None, :]
    ar, ai = slices(As.real, n_slices), slices(As.imag, n_slices)
    br, bi = slices(Bs.real, n_slices), slices(Bs.imag, n_slices)
    lv = [np.zeros((A.shape[0], B.shape[1]), dtype=np.complex128) for _ in range(3)]
    for i, j in pairs(n_slices):
        lvl = min(i + j, 2)
        lv[lvl] += (ar[i] @ br[j] - ai[i] @ bi[j]) + 1j * (ar[i] @ bi[j] + ai[i] @ br[j])
    scale = np.exp2((ea[:, None] + eb[None, :]).astype(np.float64))
    zero = (ea[:, None] == ZERO_EXP) | (eb[None, :] == ZERO_EXP)
    C = np.where(zero, 0, (lv[0] + lv[1] + lv[2]) * scale)
    return C.astype(out_dtype), lv


def error_bound(A, B, ref, n_slices=N_SLICES):
    """Per-element bound on |device result - A @ B| (A: M x K, B: K x N):
    the output rounding (2^-24 relative per component, |.| <= 2^-23 |ref|)
    plus, per real product, the dropped slice pairs of level >= n_slices and
    the slice residuals (below 2^-(7 n_slices - 1) of the row / column scales
    2^ea, 2^eb, with a factor 2 of margin), two
    real products per component and K terms, and the truncations of the small
    level-2-4 accumulator (below 2^-30 of the scales after K terms)."""
    ea = row_exponents(A).astype(np.float64)
    eb = row_exponents(B.T).astype(np.float64)
    K = A.shape[1]
    scale = np.exp2(np.minimum(ea, 4096)[:, None] + np.minimum(eb, 4096)[None, :])
    return 2.0 ** -23 * np.abs(ref) + (2.0 ** -(7 * n_slices - 3) * K + 2.0 ** -29) * scale


# ---- four fp16 slices (complex64 results, K <= 256) --------------------------

HALF_MAX_K = 256
# slice 0 of A meets slices 0 .. 3 of B, slices 1 and 2 meet 0 .. 2, slice 3 meets 0
HALF_MET = (4, 3, 3, 1)
HALF_PAIRS = [(i, j) for i in range(4) for j in range(HALF_MET[i])]


def half_bits(K, side):
    """Bits of the first slice's grid and how many more the second's has, for
    the rows of A (side 0) or the columns of B (side 1)."""
    return (8 if K <= (128 if side == 0 else 256) else 7), (8 if K <= 128 else 7)


def half_slices(x, K, side):
    """The fp16 slices of x (|x| < 1); the device holds them times 2^15, which
    is why a value below 2^-29 is a multiple of 2^-39."""
    b0, more = half_bits(K, side)
    r = np.array(x, dtype=np.float64)
    out = []
    for g in (2.0 ** b0, 2.0 ** (b0 + more)):
        out.append(np.rint(r * g) / g)
        r = r - out[-1]
    for _ in range(2):
        out.append(np.float64(np.float16(r * 2.0 ** 15)) * 2.0 ** -15)
        r = r - out[-1]
    return out


def scaled(X):
    """Rows of X times 2^-e, and e."""
    e = row_exponents(X)
    return X * np.exp2(np.where(e == ZERO_EXP, 0, -e).astype(np.float64))[:, None], e


def half_matmul(A, B):
    """C = A @ B (K <= 256) from four fp16 slices, sums in FP64: (the FP64
    value of the kept pairs, levels unscaled)."""
    K = A.shape[1]
    As, ea = scaled(A)
    Bs, eb = scaled(B.T)
    a = [half_slices(v, K, 0) for v in (As.real, As.imag)]
    b = [half_slices(v.T, K, 1) for v in (Bs.real, Bs.imag)]
    lv = [np.zeros((A.shape[0], B.shape[1]), dtype=np.complex128) for _ in range(3)]
    for i, j in HALF_PAIRS:
        lv[min(i + j, 2)] += (a[0][i] @ b[0][j] - a[1][i] @ b[1][j]) + 1j * (a[0][i] @ b[1][j] + a[1][i] @ b[0][j])
    scale = np.exp2((ea[:, None] + eb[None, :]).astype(np.float64))
    return (lv[0] + lv[1] + lv[2]) * scale, lv


def truncate24(x):
    """x rounded toward zero to FP32's 24 significant bits."""
    m, e = np.frexp(x)
    return np.ldexp(np.trunc(np.ldexp(m, 24)), e - 24)


def accumulate(A, B, half, order=None):
    """A @ B as the tensor core adds it up, unrounded: 16-term sums of exact
    products, each added to its level's accumulator and truncated, K tile by K
    tile.  ``half``: four fp16 slices, within a K tile by slice of A and of B
    from the last to the first; else five bf16 ones, within a K tile by level
    with the smallest of the rest first (``order`` "level"), or "slice" as the
    others."""
    K = A.shape[1]
    As, ea = scaled(A)
    Bs, eb = scaled(B.T)
    cut = (lambda v, side: half_slices(v, K, side)) if half else (lambda v, side: slices(v))
    a = [cut(v, 0) for v in (As.real, As.imag)]
    b = [cut(v.T, 1) for v in (Bs.real, Bs.imag)]
    order = order or ("slice" if half else "level")
    ps = (list(HALF_PAIRS) if half else [(i, j) for i in range(N_SLICES) for j in range(N_SLICES - i)])[::-1]
    if order == "level":
        ps.sort(key=lambda p: (min(p[0] + p[1], 2), -(p[0] + p[1])))
    groups = []  # (slice of A, its slices of B) in issue order
    for i, j in ps:
        if order == "slice" and groups and groups[-1][0] == i:
            groups[-1][1].append(j)
        else:
            groups.append((i, [j]))
    out = np.zeros((2, 3, A.shape[0], B.shape[1]))  # (re, im) x level
    for k in range(0, K, 16):
        t = slice(k, min(K, k + 16))
        for i, js in groups:
            for part in range(2):
                for j in js:
                    lv, bp = min(i + j, 2), b[part][j][t]
                    x = (a[0][i], -a[1][i]) if part else (a[0][i], a[1][i])
                    re, im = (x[1], x[0]) if part else (x[0], x[1])
                    out[0, lv] = truncate24(out[0, lv] + re[:, t] @ bp)
                    out[1, lv] = truncate24(out[1, lv] + im[:, t] @ bp)
    scale = np.exp2((ea[:, None] + eb[None, :]).astype(np.float64))
    return (out[0].sum(0) + 1j * out[1].sum(0)) * scale
