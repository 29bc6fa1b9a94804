"""Recordings with NaN, infinities, or values so large or small that the reference's
own sums leave the normal range: the tensor-core mode has to give what the FP32
mode gives, an error of convergence included."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from spikesorting_fullpursuit_b200 import _lib, synthetic  # noqa: E402
from spikesorting_fullpursuit_b200.parallel import binary_pursuit_parallel as bpp  # noqa: E402

pytestmark = pytest.mark.gpu


def _run(v, si, m, nmax, precision, layout=None):
    stats = []
    try:
        kw = dict(tc_layout=layout) if layout else {}
        out = bpp.binary_pursuit(v, v.dtype, si, dict(m), n_max_shift_inds=nmax, precision=precision, max_passes=40,
                                 stats=stats, **kw)
    except _lib.PursuitError as e:
        return e.code, None
    return [np.asarray(a) for a in out], stats[0]["passes"]


@pytest.mark.parametrize("layout", ["samples", "wide"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, "templates", 1e-19, 1e-17, 1e17, 1e19])
@pytest.mark.parametrize("C,K,L,nmax,overlap", [(1, 8, 100, 88, True), (16, 5, 17, 11, False), (4, 17, 64, 30, True)])
def test_same_as_fp32(C, K, L, nmax, overlap, bad, layout):
    rec = synthetic.make_recording(n_chans=C, duration_s=60 * L / 30000.0, fs=30000.0, n_templates=K, L=L,
                                   pre_fraction=0.4, rate_range=(50.0, 120.0), overlap_fraction=0.4, seed=40 + L,
                                   gain="uniform")
    si = rec.sort_info(get_adjusted_clips=True, do_overlap_recheck=overlap)
    m = rec.fresh_metrics()
    v = rec.voltage.astype(np.float32)
    if bad == "templates":
        m["templates"] = np.array(m["templates"])
        m["templates"].reshape(K, -1)[K // 2, 3] = np.nan
    elif np.isfinite(bad):
        v = (v * np.float32(bad)).astype(np.float32)
        m["templates"] = np.asarray(m["templates"]) * bad
        for k in ("template_SS", "neuron_lower_thresholds"):
            m[k] = np.asarray(m[k]) * bad * bad
    else:
        v[C // 2, v.shape[1] // 3] = bad
    with np.errstate(all="ignore"):
        exp, passes = _run(v, si, m, nmax, "fp32")
        got, passes1 = _run(v, si, m, nmax, "bf16", layout)
    assert passes == passes1
    if passes is None:
        assert got == exp
        return
    for g, e in zip(got, exp):
        assert np.array_equal(g, e, equal_nan=g.dtype.kind == "f")
