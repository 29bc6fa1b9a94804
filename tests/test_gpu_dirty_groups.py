"""Listed windows recompute only the template groups whose voltage changed, and
the wide tiles take one stream of windows per group: at one group and several,
a partly filled one, more groups than one word of bits holds, the shortest and
longest templates of the wide tiles and past them, on recordings with spikes
close together, the pursuit has to find the oracle's spikes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O  # noqa: E402
from spikesorting_fullpursuit_b200 import synthetic  # noqa: E402
from spikesorting_fullpursuit_b200.parallel import binary_pursuit_parallel as bpp  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("C,K,L,mask,windows,overlap", [
    (20, 16, 16, 4, 300, True),       # one full group, the shortest templates
    (64, 49, 31, 4, 150, True),       # a last group of one template
    (32, 530, 16, 4, 60, False),      # 34 groups: two words
    (6, 18, 190, None, 24, False),    # long templates, groups on every channel
    (4, 5, 230, None, 16, True),
])
def test_pursuit_matches_oracle(C, K, L, mask, windows, overlap, precision):
    kw = dict(n_chans=C, duration_s=windows * L / 30000.0, fs=30000.0, n_templates=K, L=L, pre_fraction=0.4,
              rate_range=(60.0, 200.0) if K < 100 else (5.0, 30.0), overlap_fraction=0.5, seed=700 + K)
    kw.update(gain="mask", mask_chans=mask) if mask else kw.update(gain="uniform")
    rec = synthetic.make_recording(**kw)
    si = rec.sort_info(get_adjusted_clips=True, do_overlap_recheck=overlap)
    nmax = min(L - 1, 60)
    exp = O.binary_pursuit_oracle(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=nmax)
    got = bpp.binary_pursuit(rec.voltage, rec.voltage.dtype, si, rec.fresh_metrics(), n_max_shift_inds=nmax,
                             precision=precision)
    assert len(exp[0]) > 0
    for g, e in zip(got, exp):
        assert np.array_equal(np.asarray(g), np.asarray(e))
