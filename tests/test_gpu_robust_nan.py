"""Robust templates of columns with NaN and infinities at the sizes where the kernel
changes its way of selecting: NaN counts as larger than every other value, and a
column of one value only, or with an infinite median, gives that."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import preprocessing as PRE  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [2, 3, 5, 31, 32, 33, 63, 64, 65, 66, 601, 4096, 4097])
def test_columns_with_nan_and_infinities(m):
    r = np.random.Generator(np.random.PCG64(m))
    p = r.permutation(m)
    x = np.zeros((m, 6), np.float32)
    x[:, 0] = np.nan
    x[:, 1] = np.where(p == 0, np.nan, p)            # 1 .. m - 1 and NaN
    x[:, 2] = p - (m - 1) / 2                        # symmetric about 0, no NaN
    x[:, 3] = np.where(p == m - 1, np.nan, p - (m - 1) / 2.0)     # NaN in the place of the largest
    x[:, 4] = np.where(p <= m // 2, np.inf, p)
    x[:, 5] = np.where(p <= m // 2, -np.inf, p)
    got = np.asarray(PRE.calculate_robust_template(x))
    # the middle of m values in steps of 1, NaN in the highest place; the values within
    # one deviation of it lie on both sides alike, and two values have a median of NaN
    # where one of them is NaN
    exp1 = (m + 1) / 2.0 if m > 2 else np.nan
    exp3 = 0.0 if m > 2 else np.nan
    # what lies within one deviation of the middle may hold one value more on one side
    assert np.isnan(got[0])
    for c, e in ((1, exp1), (2, 0.0), (3, exp3)):
        assert (np.isnan(got[c]) and np.isnan(e)) or abs(got[c] - e) <= 0.5, (c, got[c], e)
    assert got[4] == np.inf and got[5] == -np.inf
