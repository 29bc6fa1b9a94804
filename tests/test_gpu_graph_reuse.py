"""Two pursuits in the same buffers whose templates differ only in the width of
their supports: the second has to use its own rounding bounds, not those that
the first one's captured passes hold."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


class _Buffers:
    def __init__(self, C, n, K, L, nmax):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        size = ctypes.c_size_t(0)
        _lib.check(_lib.lib().fbp_pursuit_workspace_bytes(n, C, K, L, nmax, _lib.PREC_BF16_REFINE, ctypes.byref(size)))
        self.cap = 8 * (n // L + 1) + 4096
        f = lambda *s: torch.empty(*s, dtype=torch.float32, device=self.dev)  # noqa: E731
        self.v, self.T, self.tss, self.thr = f(C, n), f(K, C * L), f(K), f(K)
        self.ws = torch.empty(size.value, dtype=torch.uint8, device=self.dev)
        self.out = torch.empty(2, self.cap, dtype=torch.int32, device=self.dev)
        self.shape = (C, n, K, L, nmax)

    def pursue(self, v, T, tss, thr, layout):
        C, n, K, L, nmax = self.shape
        lib = _lib.lib()
        for d, h in ((self.v, v), (self.T, T), (self.tss, tss), (self.thr, thr)):
            d.copy_(torch.from_numpy(h))
        m, passes, st = ctypes.c_uint32(0), ctypes.c_uint32(0), _lib.StageStats()
        p = _lib.ptr
        _lib.check(lib.fbp_set_tc_layout(layout))
        try:
            _lib.check(lib.fbp_pursuit_chunk(p(self.v), n, C, p(self.T), K, L, p(self.tss), p(self.thr), nmax, 1,
                                             _lib.PREC_BF16_REFINE, 0, 1000, p(self.ws), self.ws.numel(),
                                             p(self.out[0]), p(self.out[1]), self.cap, None, ctypes.byref(m),
                                             ctypes.byref(passes), 0, ctypes.byref(st), None))
        finally:
            _lib.check(lib.fbp_set_tc_layout(_lib.TC_LAYOUT_AUTO))
        torch.cuda.synchronize()
        o = self.out[:, :m.value].cpu().numpy().view(np.uint32)
        return o, int(st.lik_refined), int(st.lik_seq_refined), int(passes.value)


@pytest.mark.parametrize("layout", [_lib.TC_LAYOUT_SAMPLES, _lib.TC_LAYOUT_WIDE])
def test_wider_templates_in_the_same_buffers(layout):
    C, K, L, nmax, n = 17, 8, 61, 60, 61 * 400
    r = np.random.Generator(np.random.PCG64(17))
    shape = np.sin(np.linspace(0, 3 * np.pi, L)) * np.hanning(L)
    wide = np.float32(2 * shape * r.uniform(0.3, 1.0, (K, C, 1)) + 0.05 * r.standard_normal((K, C, L)))
    narrow = np.zeros_like(wide)
    for k in range(K):                               # two channels each, the first and the last among them
        c = (C - 2) * k // (K - 1)
        narrow[k, c:c + 2] = wide[k, c:c + 2]
    v = r.standard_normal((C, n)).astype(np.float32) * 4
    for s in np.sort(r.choice(n - 3 * L, 250, replace=False)):
        v[:, s:s + L] += wide[r.integers(K)]

    def args(T):
        tss = np.float32(-0.5 * (T.astype(np.float64) ** 2).sum((1, 2)))
        return v, np.ascontiguousarray(T.reshape(K, -1)), tss, np.float32(0.3 * -tss)

    a, b = _Buffers(C, n, K, L, nmax), _Buffers(C, n, K, L, nmax)
    a.pursue(*args(narrow), layout)
    got, refined, seq, passes = a.pursue(*args(wide), layout)
    exp, refined1, seq1, passes1 = b.pursue(*args(wide), layout)
    _, T, tss, thr = args(wide)
    i, lab, _, _ = O.pursuit_chunk(v.copy(), T.reshape(-1), K, L, tss, thr, nmax, True)
    assert refined1 > 1000
    assert (refined, seq, passes) == (refined1, seq1, passes1)
    for o in (got, exp):
        assert np.array_equal(o[0], i) and np.array_equal(o[1], lab)
