"""Robust templates and clip covariances at the edges of their kernels' splits:
units of 64 spikes and 4096 spikes and one more, columns of equal values, with
an outlier that crowds the other values into one bin, with infinities and NaN;
templates of lengths around the covariance's tiles of 4."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import _lib  # noqa: E402
from spikesorting_fullpursuit_b200 import preprocessing as PRE  # noqa: E402

pytestmark = pytest.mark.gpu


def _median(key):          # of a sorted float array, by the rule of the mean of the middle two
    n = len(key)
    return key[n // 2] if n % 2 else key.dtype.type((key[n // 2 - 1] + key[n // 2]) * key.dtype.type(0.5))


def _robust(col):
    t = np.float32 if col.dtype == np.float32 else np.float64
    s = np.sort(col).astype(t)
    med = _median(s)
    mad = t(_median(np.sort(np.abs(s - med))) / t(0.6745))
    inner = s[(s > med - mad) & (s < med + mad)]
    r = _median(inner) if len(inner) else med
    return r if t == np.float32 else np.int16(r)


@pytest.mark.parametrize("dt", [np.float32, np.int16])
@pytest.mark.parametrize("m", [2, 3, 31, 63, 64, 65, 66, 127, 600, 601, 4096, 4097])
def test_robust_template_of_edge_sizes(m, dt):
    r = np.random.Generator(np.random.PCG64(m))
    x = (r.standard_normal((m, 7)) * 300).astype(np.float32)
    x[:, 1] = 17.0                                   # one value
    x[0, 2] = 3.0e4                                  # the rest in few bins
    x[:, 3] = r.integers(-2, 3, m)                   # ties
    x[:, 4] = np.abs(x[:, 4]) * 0.003 + 50.0
    x[:, 5] = np.where(r.random(m) < 0.5, -1000.0, 1000.0)
    x = np.round(x).astype(dt) if dt == np.int16 else x
    got = PRE.calculate_robust_template(x)
    exp = np.array([_robust(np.ascontiguousarray(x[:, c])) for c in range(x.shape[1])])
    assert np.array_equal(np.asarray(got), exp)


@pytest.mark.parametrize("bad", [np.inf, -np.inf])
def test_robust_template_with_an_infinite_value(bad):
    r = np.random.Generator(np.random.PCG64(5))
    x = r.standard_normal((201, 3)).astype(np.float32)
    x[7, 1] = bad
    got = np.asarray(PRE.calculate_robust_template(x))
    assert np.array_equal(got, np.array([_robust(np.ascontiguousarray(x[:, c])) for c in range(3)]))


@pytest.mark.parametrize("C,L,n", [(1, 1, 3), (2, 3, 33), (1, 4, 64), (3, 5, 257), (2, 9, 1000), (1, 109, 70), (2, 110, 300)])
def test_clip_covariance_of_edge_lengths(C, L, n):
    r = np.random.Generator(np.random.PCG64(L))
    clips = r.standard_normal((n, C * L)).astype(np.float32)
    tmpl = (r.standard_normal((2, C * L)) * 0.1).astype(np.float32)
    unit = r.integers(0, 2, n).astype(np.uint32)
    rows = np.sort(r.choice(n, size=max(1, n - 1), replace=False)).astype(np.int64)
    dev = torch.device("cuda", torch.cuda.current_device())
    d = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).to(dev)  # noqa: E731
    t = [d(a) for a in (clips, unit, tmpl, rows)]
    cov = torch.empty((C, L, L), dtype=torch.float64, device=dev)
    lib = _lib.lib()
    sb = lib.fbp_noise_cov_scratch_bytes(C, L)
    scratch = torch.empty(sb, dtype=torch.uint8, device=dev)
    p = _lib.ptr
    _lib.check(lib.fbp_clip_noise_covariance(p(t[0]), 0, p(t[1]), p(t[2]), p(t[3]), len(rows), C, L, p(cov),
                                             p(scratch), ctypes.c_size_t(sb), None))
    torch.cuda.synchronize()
    x = (clips[rows] - tmpl[unit[rows]]).astype(np.float64).reshape(len(rows), C, L)
    x = x - x.mean(axis=0)
    exp = np.einsum("rci,rcj->cij", x, x) / len(rows)
    scale = np.sqrt(np.einsum("rci->ci", x * x) / len(rows)) + 1e-3
    # a sum of n products, each side rounded n times, and the means
    tol = 8 * (len(rows) + 4) * 2.0 ** -53 * scale[:, :, None] * scale[:, None, :]
    got = cov.cpu().numpy()
    assert np.all(np.abs(got - exp) <= tol)
