"""The reference detector's block statistics over the data that decide how they are formed: sums
that are exact whatever their order, sums whose chain rounds, data that only the chains as written
can settle (a mean far above the rms, values of very different sizes, zeros, infinities), chunk
counts and lengths off the kernels' tiles.  Equal to the oracle's chains bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _series(kind, ndms, nsamp, seed):
    rng = np.random.default_rng(seed)
    y = rng.standard_normal((ndms, nsamp), dtype=np.float32) * np.float32(16.0)
    if kind == "offset":      # an 8-bit block's sums: mean far above the rms
        y = np.rint(y * 64 + 524288).astype(np.float32)
    elif kind == "integers":
        y = np.rint(y)
    elif kind == "spread":    # tiny and large values in one chunk
        y[:, ::97] *= np.float32(1e-6)
        y[:, ::1013] *= np.float32(3e4)
    elif kind == "zeros":
        y[:, : nsamp // 2] = 0.0
    elif kind == "small":
        y *= np.float32(1e-12)
    elif kind == "drift":
        y += np.linspace(-300, 500, nsamp, dtype=np.float32)[None, :]
    elif kind == "inf":
        y[0, nsamp // 3] = np.inf
    y[ndms // 2, nsamp // 4:nsamp // 4 + 6] += np.float32(2000.0)
    return y


@pytest.mark.parametrize("kind", ["noise", "offset", "integers", "spread", "zeros", "small",
                                  "drift", "inf"])
@pytest.mark.parametrize("ndms,nsamp", [(1, 5), (3, 701), (5, 6553), (7, 9363), (64, 40001),
                                        (200, 16384)])
def test_statistics_equal_the_chains(lib, orc, cuda, kind, ndms, nsamp):
    import mdsm_gb300 as m
    y = _series(kind, ndms, nsamp, ndms + nsamp)
    cands, mean, rms, n = m.ref_detect_device(cuda.from_numpy(y).cuda(), 2.0, 0.5, 5.0)
    with np.errstate(all="ignore"):
        (dm, samp, snr), om, orms = orc.ref_detect(y, 2.0, 0.5, 5.0)
    assert np.array_equal([mean, rms], [om, orms], equal_nan=True)
    assert n == len(dm)
    k = np.lexsort((samp, dm))
    assert np.array_equal(cands["dm_idx"], dm[k]) and np.array_equal(cands["sample"], samp[k])
    assert np.array_equal(cands["snr"], snr[k], equal_nan=True)
