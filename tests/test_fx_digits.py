"""The exact-digit DST of the FP64 path (mw3_fx.cu) on the CPU: the same fixed-point
vectors, base-256 digits, groups and 64-bit sum in integer numpy, against a
long-double product and beside plain FP64."""
import numpy as np
import pytest

ND = 7


def _digits(X):
    """Signed base-256 digits, the largest first; the first takes what is left."""
    X = X.astype(np.int64).copy()
    d = np.zeros((ND,) + X.shape, np.int64)
    for i in range(ND - 1, 0, -1):
        d[i] = ((X + 128) & 255) - 128
        X = (X - d[i]) >> 8
    d[0] = X
    return d


def _fixed(x, ef, sh):
    """round(x 2^(57 - E)) (half away from zero), E = ef - 1022, one bit less for sh = 3."""
    bits = np.abs(x).view(np.int64)
    ex = bits >> 52
    m = (bits & ((1 << 52) - 1)) | np.where(ex > 0, 1 << 52, 0)
    r = np.minimum(np.where(ef - np.maximum(ex, 1) < 0, 63, ef - np.maximum(ex, 1)), 63)
    v = ((m << sh) + ((np.int64(1) << r) >> 1)) >> r
    return np.where(np.signbit(x), -v, v)


def _sine_ld(n):
    k = np.arange(1, n + 1)
    m = np.outer(k, k) % (2 * (n + 1))
    return 2 * np.sin(np.longdouble(np.pi) * 0 + _pi_ld() * m.astype(np.longdouble) / (n + 1))


def _pi_ld():
    return np.longdouble("3.141592653589793238462643383279502884")


def _product(S, x, sh):
    """sum_k S[i][k] x[..][k] as the kernel forms it."""
    ef = (np.abs(x).max(-1).view(np.int64) >> 52)[..., None]
    return _from_fixed(S, _fixed(x, ef, sh), ef, sh)


def _from_fixed(S, X, ef, sh):
    s = _digits(np.rint(S * np.longdouble(2.0) ** 54).astype(np.int64))
    d = _digits(X)
    a = [sum(d[j] @ s[g - j].T for j in range(g + 1)) for g in range(ND)]
    for g in range(5):
        assert np.abs(a[g]).max() <= 1 << 24          # what an FP32 accumulator holds exactly
    H = (a[0] << 24) + (a[1] << 16) + (a[2] << 8) + a[3]
    L = (a[4] << 16) + (a[5] << 8) + a[6]
    mag = np.maximum(np.abs(H), 1)
    z = np.minimum(24, 62 - np.frexp(mag.astype(np.float64))[1])     # (H < 2^53 here: exact)
    V = (H << z) + (L >> (24 - z))
    return np.ldexp(V.astype(np.float64), (ef - 1061 + 4 - sh - z).astype(np.int32))


def _folded(x, n):
    """The transform of length n through sums and differences of mirrored entries."""
    S, h = _sine_ld(n), (n + 1) // 2
    ef = (np.abs(x).max(-1).view(np.int64) >> 52)[..., None]
    sh = 3 if n < 480 else 2                           # as the tables' own bound asks for
    X = _fixed(x, ef, sh)
    lo, hi = X[..., :h], X[..., ::-1][..., :h]
    even, odd = lo + hi, lo - hi
    if n % 2:
        even[..., h - 1] = lo[..., h - 1]
    y = np.empty(x.shape)
    y[..., 0::2] = _from_fixed(S[0::2, :h], even, ef, sh)
    y[..., 1::2] = _from_fixed(S[1::2, :h], odd, ef, sh)
    return y


def _inputs(n, kind, rng):
    k = np.arange(n)
    if kind == "normal":
        return rng.normal(size=(8, n))
    if kind == "packet":
        c = rng.uniform(0.2, 0.8, 8)[:, None] * n
        return np.exp(-((k - c) / (0.06 * n)) ** 2) * np.cos(0.9 * k + c) * 10.0 ** rng.uniform(-12, 3, (8, 1))
    if kind == "wide":                                 # entries over 40 decades
        return rng.normal(size=(8, n)) * 10.0 ** rng.uniform(-40, 0, (8, n))
    return np.ones((8, n)) * np.array([1, -1, 1 - 2.0 ** -53, 255 / 256, 3, 1e-300, 1e300, 0.1])[:, None]


@pytest.mark.parametrize("kind", ["normal", "packet", "wide", "flat"])
@pytest.mark.parametrize("n,folded", [(5, False), (16, False), (60, False), (127, False), (128, False),
                                      (41, True), (192, True), (255, True), (256, True), (512, True)])
def test_digit_products_are_as_exact_as_fp64(n, folded, kind):
    rng = np.random.default_rng([n, len(kind)])
    x = _inputs(n, kind, rng)
    S = _sine_ld(n)
    exact = x.astype(np.longdouble) @ S.T
    y = _folded(x, n) if folded else _product(S, x, 4)
    plain = x @ S.astype(np.float64).T
    big = np.abs(x).max(-1, keepdims=True)
    err, ref = np.abs(y - exact) / big, np.abs(plain - exact) / big
    # rounding of x (2^(E-56) at most) and of S (2^-55): n terms of 2^-54; the groups left out:
    # 6 digit pairs of at most 2^14 a term, 2^-56 of the top pair; the 62-bit sum and the result
    assert np.all(err <= n * 2.0 ** -50 + 2.0 ** -52 * np.abs(exact / big))
    rms = np.sqrt((err.astype(float) ** 2).mean())
    assert rms <= max(1.5 * np.sqrt((ref.astype(float) ** 2).mean()), np.sqrt(n) * 2.0 ** -53)
