"""The FP32 overlap tables with fewer tiles than a block of 128 threads takes,
and more than a block of 256: the pursuit has to find the
oracle's spikes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import synthetic  # noqa: E402
from spikesorting_fullpursuit_b200.parallel import binary_pursuit_parallel as bpp  # noqa: E402

pytestmark = pytest.mark.gpu


# tiles of 8 shifts x 8 templates
@pytest.mark.parametrize("C,K,L,nmax", [(2, 32, 61, 60), (2, 33, 63, 63), (1, 60, 33, 66), (1, 130, 33, 64)])   # 64, 80, 136, 289
def test_pursuit_matches_oracle(C, K, L, nmax):
    rec = synthetic.make_recording(n_chans=C, duration_s=60 * L / 30000.0, fs=30000.0, n_templates=K, L=L,
                                   pre_fraction=0.4, rate_range=(10.0, 40.0), overlap_fraction=0.4, seed=900 + K,
                                   gain="uniform")
    si = rec.sort_info(get_adjusted_clips=True)
    exp = O.binary_pursuit_oracle(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=nmax)
    got = bpp.binary_pursuit(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=nmax,
                             precision="fp32")
    assert len(exp[0]) > 0
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g), np.asarray(e))
