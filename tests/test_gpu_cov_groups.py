"""Clip covariances of short templates, whose blocks have several groups of threads,
around the lengths at which the number of groups changes, against float64 numpy."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.int16])
@pytest.mark.parametrize("C,L,n", [(1, 1, 1), (2, 4, 33), (4, 16, 1000), (1, 28, 31), (3, 31, 515), (1, 44, 65), (2, 57, 257),
                                   (1, 60, 40), (1, 61, 40)])
def test_covariance_of_grouped_blocks(C, L, n, dtype):
    r = np.random.Generator(np.random.PCG64(100 * L + n))
    clips = (300 * r.standard_normal((n + 1, C * L))).astype(dtype)
    tmpl = (30 * r.standard_normal((2, C * L))).astype(dtype)
    unit = r.integers(0, 2, n + 1).astype(np.uint32)
    rows = np.sort(r.choice(n + 1, size=n, replace=False)).astype(np.int64)
    dev = torch.device("cuda", torch.cuda.current_device())
    t = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).to(dev) for a in (clips, unit, tmpl, rows)]
    cov = torch.empty((C, L, L), dtype=torch.float64, device=dev)
    lib, p = _lib.lib(), _lib.ptr
    sb = lib.fbp_noise_cov_scratch_bytes(C, L)
    scratch = torch.empty(sb, dtype=torch.uint8, device=dev)
    _lib.check(lib.fbp_clip_noise_covariance(p(t[0]), 0 if dtype == np.float32 else 1, p(t[1]), p(t[2]), p(t[3]), n, C, L,
                                             p(cov), p(scratch), ctypes.c_size_t(sb), None))
    torch.cuda.synchronize()
    x = (clips[rows] - tmpl[unit[rows]]).astype(np.float64).reshape(n, C, L)
    x = x - x.mean(axis=0)
    exp = np.einsum("rci,rcj->cij", x, x) / n
    scale = np.sqrt(np.einsum("rci->ci", x * x) / n) + 300 * 2.0 ** -20
    # sums of n products, each side rounded n times, and the means
    tol = 8 * (n + 4) * 2.0 ** -53 * scale[:, :, None] * scale[:, None, :]
    got = cov.cpu().numpy()
    assert np.all(np.abs(got - exp) <= tol)
    assert np.all(np.abs(got - got.transpose(0, 2, 1)) <= tol)
