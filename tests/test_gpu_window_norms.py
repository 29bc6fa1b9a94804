"""The window norms behind the tensor-core likelihood's error bound come from the
float32 samples: a recording whose second half is larger by less than fp16
resolves has bounds larger by that factor there."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [_lib.TC_LAYOUT_SAMPLES, _lib.TC_LAYOUT_WIDE])
@pytest.mark.parametrize("C,K,L", [(3, 3, 16), (9, 18, 61), (1, 2, 190), (2, 2, 260)])
def test_norms_resolve_what_fp16_does_not(C, K, L, layout):
    lib, dev = _lib.lib(), torch.device("cuda", torch.cuda.current_device())
    r = np.random.Generator(np.random.PCG64(L))
    n = (12000 + 8 * L) // (16 * L) * 16 * L         # halves that start at multiples of 8
    grow = np.float32(1.0 + 0.95 * 2.0 ** -11)       # rounds to 1 in fp16
    v = np.where(r.random((C, n)) < 0.5, np.float32(-1), np.float32(1))
    v[:, n // 2:] *= grow
    T = np.float32(1e-2 * r.standard_normal((K, C * L)) / np.sqrt(C * L))
    tss = np.float32(-0.5 * (T.astype(np.float64) ** 2).sum(1))
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (v, T, tss)]
    size = ctypes.c_size_t(0)
    _lib.check(lib.fbp_pursuit_workspace_bytes(n, C, K, L, 0, _lib.PREC_BF16_REFINE, ctypes.byref(size)))
    ws = torch.empty(size.value, dtype=torch.uint8, device=dev)
    out = torch.zeros(2, K, n, dtype=torch.float32, device=dev)
    p = _lib.ptr
    _lib.check(lib.fbp_set_tc_layout(layout))
    try:
        _lib.check(lib.fbp_tc_likelihood_bounds(p(d[0]), n, C, p(d[1]), K, L, p(d[2]), p(ws), ws.numel(), p(out[0]),
                                                p(out[1]), None))
    finally:
        _lib.check(lib.fbp_set_tc_layout(_lib.TC_LAYOUT_AUTO))
    torch.cuda.synchronize()
    approx, E = out.cpu().numpy().astype(np.float64)
    R = E - 2.0 ** -22 * np.abs(approx)              # what is left is proportional to the norm, but for kappa_s |SS/2|
    a = R[:, 2 * L:n // 2 - 2 * L]
    b = R[:, n // 2 + 2 * L:n - 3 * L]
    # kappa_s |SS/2| against kappa ||t|| ||window||, with kappa >= 2^-10 and ||window|| = sqrt(C L): less than
    # (C L + 6) 2^-24 1.1 ||t|| / (2^-9 sqrt(C L)); the rest are float32 roundings (C L products and sums)
    tol = (C * L + 6) * 2.0 ** -14 * 1e-2 / np.sqrt(C * L) + (C + 40) * 2.0 ** -23
    assert tol < 0.1 * (float(grow) - 1)
    for m in range(8):                               # positions alike within the blocks of 8
        ra, rb = a[:, m::8], b[:, m::8]
        assert np.all(ra > 0) and np.all(rb > 0)
        ratio = rb.mean(1) / ra.mean(1)
        assert np.all(np.abs(ratio / float(grow) - 1) <= tol), (m, ratio)
