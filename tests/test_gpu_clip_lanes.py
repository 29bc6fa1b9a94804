"""Clips of every length around the numbers of lanes that copy one, in both data
types, for one and several channels, against numpy."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.int16])
@pytest.mark.parametrize("W", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 130])
def test_clips_of_every_length(W, dtype):
    r = np.random.Generator(np.random.PCG64(W))
    C, n, count, first = 5, 3000, 517, 2
    v = r.integers(-3000, 3000, (C, n)).astype(dtype)
    chans = np.array([4, 0, 3], np.int64)
    ev = r.integers(200, n - 200, first + count).astype(np.int64)
    w0 = -(W // 3)
    dev = torch.device("cuda", torch.cuda.current_device())
    d = [torch.from_numpy(x).to(dev) for x in (v, chans, ev)]
    for nch in (1, 3):
        out = torch.full((count, nch * W + 1), 7, dtype=d[0].dtype, device=dev)     # a column to spare
        flat = out.view(-1)
        _lib.check(_lib.lib().fbp_get_clips(_lib.ptr(d[0]), 0 if dtype == np.float32 else 1, n, C, _lib.ptr(d[1]), nch,
                                            _lib.ptr(d[2]), first, count, w0, w0 + W, _lib.ptr(flat), None))
        torch.cuda.synchronize()
        exp = v[chans[:nch]][:, ev[first:, None] + w0 + np.arange(W)].transpose(1, 0, 2).reshape(-1)
        got = flat.cpu().numpy()
        assert np.array_equal(got[:exp.size], exp)
        assert np.all(got[exp.size:] == 7)
