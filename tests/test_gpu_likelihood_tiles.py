"""The FP32 likelihood at the edges of its tiles (64 or 128 samples), of the
steps staged at a time (256) and of its groups of 16 templates: bit for bit the
oracle's, window by window."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,K,L", [(1, 1, 1), (9, 16, 2), (17, 17, 3), (12, 15, 5), (3, 33, 63), (2, 16, 64), (2, 4, 65),
                                   (3, 5, 127), (2, 18, 128), (2, 3, 129), (1, 16, 256), (2, 5, 257), (2, 17, 515)])
def test_likelihood_bit_exact_at_tile_edges(C, K, L):
    r = np.random.Generator(np.random.PCG64(C * 1000 + L))
    n = 9 * L + L // 2 + 1
    v = r.standard_normal((C, n)).astype(np.float32)
    T = (r.standard_normal((K, C * L)) * 0.7).astype(np.float32)
    tss = np.float32(-0.5 * np.sum(T.astype(np.float64) ** 2, axis=1))
    W = (n + L - 1) // L
    win = np.sort(r.choice(W, size=max(1, W * 2 // 3), replace=False)).astype(np.uint32)
    Lk0 = r.standard_normal((K, n)).astype(np.float32)
    exp = Lk0.copy()
    O.stage_full_likelihood(v, T.reshape(-1), K, L, tss, win, exp)
    dev = torch.device("cuda", torch.cuda.current_device())
    t = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).to(dev)
         for a in (v, T, tss, win, np.array([len(win)], np.uint32), Lk0)]
    p = [_lib.ptr(x) for x in t]
    lib = _lib.lib()
    _lib.check(lib.fbp_compute_full_likelihood(p[0], n, C, p[1], K, L, p[2], p[3], p[4], W, p[5], 0, None))
    torch.cuda.synchronize()
    assert np.array_equal(t[5].cpu().numpy().view(np.uint32), exp.view(np.uint32))
