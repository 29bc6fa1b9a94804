"""Likelihoods of windows that a pass does not list keep, as in the reference,
the values of the voltage they were computed from, in the tensor-core mode
too: after a pursuit with spikes moved by the overlap recheck the stored
likelihoods of both modes agree to the tensor-core rounding bound."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import _lib, synthetic  # noqa: E402

pytestmark = pytest.mark.gpu

QUIET = 8                                            # leading windows without spikes


def _pursuit(v, T, tss, thr, K, L, nmax, prec, layout):
    """The chunk's likelihood buffer after the pursuit, found in the workspace
    by the first entries of template 0, which no spike changes."""
    lib = _lib.lib()
    C, n = v.shape
    dev = torch.device("cuda", torch.cuda.current_device())
    d = [torch.from_numpy(a).to(dev) for a in (v, T, tss, thr)]
    size = ctypes.c_size_t(0)
    _lib.check(lib.fbp_pursuit_workspace_bytes(n, C, K, L, nmax, prec, ctypes.byref(size)))
    ws = torch.zeros(size.value, dtype=torch.uint8, device=dev)
    cap = 8 * (n // L + 1) + 4096
    out = torch.empty(2, cap, dtype=torch.int32, device=dev)
    m, passes = ctypes.c_uint32(0), ctypes.c_uint32(0)
    _lib.check(lib.fbp_set_tc_layout(layout))
    try:
        _lib.check(lib.fbp_pursuit_chunk(_lib.ptr(d[0]), n, C, _lib.ptr(d[1]), K, L, _lib.ptr(d[2]), _lib.ptr(d[3]), nmax,
                                         1, prec, 0, 1000, _lib.ptr(ws), ws.numel(), _lib.ptr(out[0]), _lib.ptr(out[1]),
                                         cap, None, ctypes.byref(m), ctypes.byref(passes), 0, None, None))
    finally:
        _lib.check(lib.fbp_set_tc_layout(_lib.TC_LAYOUT_AUTO))
    torch.cuda.synchronize()
    f = ws[:size.value // 256 * 256].cpu().numpy().view(np.float32)
    first = np.zeros((K, n), np.float32)
    W = (n + L - 1) // L
    O.stage_full_likelihood(v, T.reshape(-1), K, L, tss, np.arange(W, dtype=np.uint32), first)
    q = (QUIET - 2) * L
    tol = 1e-2 * np.abs(first[0, :q]).max()
    at = [o for o in range(0, len(f) - K * n, 64) if np.all(np.abs(f[o:o + q] - first[0, :q]) <= tol)]
    assert len(at) == 1
    return f[at[0]:at[0] + K * n].reshape(K, n), int(m.value), int(passes.value)


# Templates whose threshold is out of reach leave positive likelihoods in windows that
# are not listed any more; spikes found by the overlap recheck lie up to 1.5 windows away
# from their own.  In the first case an argmax settles an entry, a moved spike then
# changes its voltage, and two passes after it was settled a neighbour reads it again.
@pytest.mark.parametrize("layout", ["samples", "wide"])
@pytest.mark.parametrize("windows,factors,seed", [
    (540, [0.3, 2.0, 1.0, 8.0, 1.0, 1.0], 105984),
    (725, [1.0, 1.0, 2.0, 0.05, 0.05, 8.0, 8.0, 2.0, 8.0, 0.05, 8.0, 1.0], 106103),
])
def test_stored_likelihoods_of_both_modes_agree(windows, factors, seed, layout):
    C, K, L, nmax = 1, len(factors), 20, 30
    rec = synthetic.make_recording(n_chans=C, duration_s=windows * L / 30000.0, fs=30000.0, n_templates=K, L=L,
                                   pre_fraction=0.4, rate_range=(8000.0 / 3 / K, 8000.0 / K), overlap_fraction=0.6,
                                   seed=seed, gain="uniform")
    quiet = np.random.Generator(np.random.PCG64(1)).standard_normal((C, QUIET * L)).astype(np.float32) * 1e-3
    v = np.ascontiguousarray(np.concatenate([quiet, rec.voltage.astype(np.float32)], axis=1))
    m = rec.fresh_metrics()
    T = np.ascontiguousarray(np.float32(m["templates"]).reshape(K, -1))
    tss = np.ascontiguousarray(np.float32(-0.5 * m["template_SS"]))
    thr = np.ascontiguousarray(np.float32(0.5 * np.asarray(m["template_SS"]) * np.array(factors)))
    exact, m0, p0 = _pursuit(v, T, tss, thr, K, L, nmax, _lib.PREC_FP32, _lib.TC_LAYOUT_AUTO)
    got, m1, p1 = _pursuit(v, T, tss, thr, K, L, nmax, _lib.PREC_BF16_REFINE,
                           _lib.TC_LAYOUT_WIDE if layout == "wide" else _lib.TC_LAYOUT_SAMPLES)
    assert (m0, p0) == (m1, p1) and p0 >= 4
    # operands rounded to fp16 (2^-10 of ||t|| ||window||), sums of C L terms in
    # float32; a window's norm grows by no more than a factor of 2 beside its
    # neighbours', whose spikes are subtracted from it
    wn = np.sqrt(np.lib.stride_tricks.sliding_window_view((v.astype(np.float64) ** 2).sum(0), L).sum(1))
    wn = np.pad(np.pad(wn, (0, L - 1)), 2 * L, mode="edge")
    wn = np.lib.stride_tricks.sliding_window_view(wn, 4 * L + 1).max(1)
    tn = np.sqrt((T.astype(np.float64) ** 2).sum(1))[:, None]
    tol = 2 * tn * wn * (2.0 ** -10 + 4 * C * L * 2.0 ** -24) + 1e-6 * np.abs(tss)[:, None]
    bad = np.argwhere(~(np.abs(got.astype(np.float64) - exact) <= tol))
    assert len(bad) == 0, (len(bad), [(tuple(b), got[tuple(b)], exact[tuple(b)]) for b in bad[:4]])
