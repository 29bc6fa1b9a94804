"""Shapes whose workspace has no room for the buffers that only save time: the dirty
bits of the FP32 mode (more than 1,024 templates, shifts above two templates), the
lag bounds of the overlap scan (many templates, a short recording).  The pursuit has
to find the oracle's spikes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import synthetic  # noqa: E402
from spikesorting_fullpursuit_b200.parallel import binary_pursuit_parallel as bpp  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("C,K,L,nmax,windows,overlap", [
    (2, 1100, 8, 20, 60, False),
    (2, 530, 8, 20, 60, False),
    (3, 20, 16, 40, 80, True),
    (24, 300, 61, 60, 12, True),
])
def test_pursuit_matches_oracle(C, K, L, nmax, windows, overlap, precision):
    kw = dict(n_chans=C, duration_s=windows * L / 30000.0, fs=30000.0, n_templates=K, L=L, pre_fraction=0.4,
              rate_range=(2000.0 / K, 6000.0 / K), overlap_fraction=0.4, seed=60 + K)
    kw.update(gain="mask", mask_chans=4) if C > 20 else kw.update(gain="uniform")
    rec = synthetic.make_recording(**kw)
    si = rec.sort_info(get_adjusted_clips=True, do_overlap_recheck=overlap)
    exp = O.binary_pursuit_oracle(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=nmax)
    got = bpp.binary_pursuit(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=nmax,
                             precision=precision)
    assert len(exp[0]) > 0
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g), np.asarray(e))
