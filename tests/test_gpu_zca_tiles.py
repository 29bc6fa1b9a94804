"""The whitening kernels at the edges of their tiles (32 channels, 64 samples
a step, sample ranges of 4096 and more) against numpy in float64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import preprocessing as PRE  # noqa: E402

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _masks(v, thr, cushion):
    over = np.abs(v.astype(np.float64)) > 0.9 * thr[:, None]
    out = over.copy()
    for c in range(v.shape[0]):
        for s in np.nonzero(over[c])[0]:
            out[c, max(0, s - cushion):s + cushion + 1] = True
    return out


@pytest.mark.parametrize("C,n,dtype,special", [
    (1, 63, np.float32, False), (31, 64, np.float32, False), (32, 4097, np.float32, False),
    (33, 5000, np.int16, False), (65, 8255, np.float32, False), (5, 4300, np.float32, True)])
def test_zca_covariance_and_product(C, n, dtype, special):
    r = np.random.Generator(np.random.PCG64(C * 1000 + n))
    v = r.standard_normal((C, n)) * 100.0 + r.uniform(-20, 20, (C, 1))
    v = v.astype(dtype)
    thr = np.full(C, 350.0)
    if special:                      # a value that is not finite, where other channels are masked and where not
        v[0, 100], v[1, 100], v[2, 200] = np.inf, 400.0, -np.inf
        thr[2] = np.inf              # channel 2 keeps its infinity
        v[3, 195:205] = 400.0
    m = _masks(v, thr, 3)
    got = PRE.zca_covariance(v, thr, 3)
    x = v.astype(np.float64)
    for i in range(C):
        for j in range(i, C):
            ok = ~m[i] & ~m[j]
            cnt = np.sum(ok)
            with np.errstate(invalid="ignore"):
                if i == j:
                    terms = (x[i, ok] - np.mean(x[i, ok])) ** 2
                else:
                    terms = x[i, ok] * x[j, ok]
                exp = np.sum(terms) / (cnt - 1.0)
            if not np.isfinite(exp):
                assert not np.isfinite(got[i, j]), (i, j)
                continue
            # any order of n additions and one rounding a product, on both sides; the mean's own error likewise
            tol = 8.0 * n * U * (np.sum(np.abs(terms)) + np.sum(np.abs(x[i, ok]))) / (cnt - 1.0)
            assert abs(got[i, j] - exp) <= tol and got[i, j] == got[j, i], (i, j, got[i, j], exp)
    if special:
        return
    Z = r.standard_normal((C, C))
    out = PRE.zca_apply(Z, v)
    exp = Z @ x
    tol = 2.0 * C * U * (np.abs(Z) @ np.abs(x))
    if dtype == np.float32:
        assert np.all(np.abs(out - exp) <= tol + 2.0 ** -24 * np.abs(exp) * (1 + 1e-9))
    else:
        lo, hi = np.trunc(exp - tol), np.trunc(exp + tol)
        small = np.abs(exp) < 32767
        assert np.all(((out == lo) | (out == hi))[small])
