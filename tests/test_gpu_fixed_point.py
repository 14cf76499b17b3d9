"""The FP64 transforms run in 64-bit fixed point on the integer pipe (csrc/sdd_fixed.cuh): every radix and odd
length against dense sums in extended precision, rows of very different magnitude sharing one complex
transform, the ends of the exponent range, and rows with an infinity or a NaN.

Tolerance.  A row is rounded to 60 bits below a power of two E with sum|x| <= E <= 4 sum|x| (the bound is a
power of two above a sum formed with a relative slack below 1/16).  Rounding the inputs (variance 1/12 ulp^2
each) and the operations of up to 8 stages (below 1/2 ulp^2 each, carried on by the remaining stages) leaves
an error of about sqrt(2 P) ulp; 16 sqrt(P) 2^-60 E <= 16 sqrt(P) 2^-58 sum|x| is more than ten times that, plus
one rounding of the result to a double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _dense(kind, x, n):
    """The library's transforms as sums (Transforms.py:73-129), extended precision; x (rows, n_in)."""
    n_in = x.shape[1]
    L = n if kind.startswith("I") else n_in
    i = np.arange(L).astype(LD)
    pi = LD("3.14159265358979323846264338327950288")
    th = pi * (2 * i + 1) / (2 * LD(L))
    k = np.arange(n_in if kind.startswith("I") else n)
    c = np.cos(np.outer(k, th)) if kind.endswith("CT") else np.sin(np.outer(k, th))
    x = x.astype(LD)
    if kind == "IDST":
        c[0] = 0
        c[n_in:] = 0
    if kind.startswith("I"):
        return x @ c
    y = (x @ c.T) * (LD(2) / L)
    if kind == "DCT":
        y[:, 0] /= 2
    return y


@pytest.mark.parametrize("L", [2, 3, 4, 5, 6, 7, 12, 15, 21, 35, 45, 64, 96, 135, 225, 384, 405, 486, 735, 810])
def test_transforms_to_the_fixed_point_bound(cuda, L):
    from spectraldoublediffusiveconvection_gb300 import Transforms as T
    rng = np.random.default_rng(L)
    x = rng.standard_normal((7, L))
    x[1] *= np.exp(-np.arange(L) / 5.0)
    x[2] *= 1e-9                       # next to row 3 in one complex transform
    x[3] *= 1e9
    x[4] *= 1e-290
    x[5] *= 1e290
    x[6] = 0.0
    x[6, L // 2] = 1.0
    for kind in ("DCT", "DST", "IDCT", "IDST"):
        y = np.asarray(getattr(T, kind)(x.copy(), n=L))
        ref = _dense(kind, x, L)
        l1 = np.abs(x).sum(axis=1, keepdims=True)
        scale = 1.0 if kind.startswith("I") else 2.0 / L
        tol = 16 * np.sqrt(L) * 2.0 ** -58 * l1 * scale + 2.0 ** -52 * np.abs(ref).astype(float)
        assert np.all(np.abs((y - ref).astype(float)) <= tol), kind


def test_non_finite_rows_stay_in_their_pair(cuda):
    from spectraldoublediffusiveconvection_gb300 import Transforms as T
    x = np.random.default_rng(3).standard_normal((8, 48))
    good = np.asarray(T.IDCT(x.copy(), n=48))
    x[2, 5] = np.nan
    x[5, 7] = np.inf
    y = np.asarray(T.IDCT(x.copy(), n=48))
    assert np.isnan(y[2]).all() and np.isnan(y[5]).all()
    for r in (0, 1, 6, 7):
        assert np.array_equal(y[r], good[r])
