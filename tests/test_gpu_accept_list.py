"""The stage entry of the accept step goes by its window list: active windows that
are not listed are left out, and windows that are listed are looked at."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("W", [9, 4097, 66 * 4096])
def test_accept_follows_the_window_list(W, noalloc):
    L, K, dev = 3, 4, torch.device("cuda", torch.cuda.current_device())
    n = W * L
    rng = np.random.Generator(np.random.PCG64(W))
    lib = _lib.lib()
    Wp, wb = W + 4, lib.fbp_window_u8_bytes(W)
    thr = np.array([1.0, 2.0, 3.0, 4.0], np.float32)
    active = np.zeros(wb, np.uint8)
    active[:W] = rng.random(W) < 0.7
    listed = rng.random(W) < 0.5                     # neither within the active windows nor around them
    win = np.nonzero(listed)[0].astype(np.uint32)
    lab = rng.integers(0, K, Wp).astype(np.uint32)
    idx = (np.arange(Wp, dtype=np.int64) * L + rng.integers(-1, L + 1, Wp)).clip(0).astype(np.uint32)
    ll = rng.uniform(0, 5, Wp).astype(np.float32)
    ovr = np.zeros(wb, np.uint8)
    ovr[:W] = rng.random(W) < 0.1
    t = {k: torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).to(dev)
         for k, v in dict(lab=lab, idx=idx, ll=ll, ovr=ovr, flags=active, active=active, win=win, thr=thr).items()}
    p = _lib.ptr
    st = _lib.WindowState(*[p(t[k]) for k in ("idx", "lab", "ll", "idx", "lab", "flags", "ovr")])
    out = [torch.full((Wp,), -1, dtype=torch.int32, device=dev) for _ in range(3)]
    has = torch.full((wb,), 7, dtype=torch.uint8, device=dev)
    fout = torch.zeros(wb, dtype=torch.uint8, device=dev)
    nwin = torch.tensor([len(win)], dtype=torch.int32, device=dev)
    nspk = torch.zeros(1, dtype=torch.int32, device=dev)
    scan = torch.empty(lib.fbp_scan_scratch_bytes(W), dtype=torch.uint8, device=dev)
    head = (n, 1, L, p(t["thr"]), p(t["win"]), p(nwin), len(win), ctypes.byref(st), p(t["active"]))
    tail = (p(fout), p(out[0]), p(out[1]), p(out[2]), p(nspk))
    for _ in range(2):                               # the second call finds the first one's scratch
        if noalloc:
            _lib.check(lib.fbp_binary_pursuit_accept_noalloc(*head, *tail, None))
        else:
            _lib.check(lib.fbp_binary_pursuit_accept(*head, p(has), *tail, p(scan), None))
    torch.cuda.synchronize()
    w = np.arange(W)
    ok = (w + 1) * L < n - L
    l_, i_, m_ = np.where(ok, lab[:W], 0), np.where(ok, idx[:W], 0), np.where(ok, ll[:W], 0)
    o = ovr[:W] == 1
    exp = np.nonzero(listed & ((m_ > thr[l_]) | o) & (((i_ >= w * L) & (i_ < (w + 1) * L)) | o))[0]
    m = int(nspk.item())
    assert m == len(exp)
    assert np.array_equal(out[2].cpu().numpy()[:m], exp)
    assert np.array_equal(out[0].cpu().numpy()[:m].view(np.uint32), i_[exp])
    assert np.array_equal(out[1].cpu().numpy()[:m].view(np.uint32), l_[exp])
