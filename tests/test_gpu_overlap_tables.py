"""The fast overlap recheck's template tables at the sizes where their kernel
changes its staging: both templates' channels in shared memory for one or two
blocks per SM, or too many channels for it, and pairs of templates without a
common channel.  The pursuit has to find the oracle's spikes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import synthetic  # noqa: E402
from spikesorting_fullpursuit_b200.parallel import binary_pursuit_parallel as bpp  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("C,K,L,mask", [
    (1, 2, 16, None),        # the smallest
    (3, 5, 33, None),        # one lag row past a warp
    (96, 4, 101, None),      # more channels than shared memory holds beside the table
    (40, 4, 90, None),       # one block per SM
    (48, 9, 31, 16),         # supports that touch, overlap or lie apart
])
def test_pursuit_matches_oracle(C, K, L, mask, precision):
    kw = dict(n_chans=C, duration_s=0.06 + 40 * L / 30000.0, fs=30000.0, n_templates=K, L=L, pre_fraction=0.4,
              rate_range=(80.0, 160.0), overlap_fraction=0.4, seed=500 + C)
    kw.update(gain="mask", mask_chans=mask) if mask else kw.update(gain="uniform")
    rec = synthetic.make_recording(**kw)
    si = rec.sort_info(get_adjusted_clips=True)
    exp = O.binary_pursuit_oracle(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=L - 1)
    got = bpp.binary_pursuit(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=L - 1,
                             precision=precision)
    assert len(exp[0]) > 0
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g), np.asarray(e))
