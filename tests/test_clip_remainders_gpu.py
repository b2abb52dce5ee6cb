"""The float clip and the detector's block statistics on samples whose sums cancel down to remainders far
below the samples themselves, beside others of many sizes: the same double sums, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows():
    rows = []
    for n, pairs, put in (
            (64, 32, [(20, 2.0 ** -42), (21, -2.0 ** -42), (22, 0.0), (23, 0.0), (62, 2.0 ** -68),
                      (63, 0.0)]),
            (1024, 16, [(40, 2.0 ** -43), (60, 2.0 ** -70)]),
            (1024, 16, [(40, 2.0 ** -43), (60, 2.0 ** -70), (70, -2.0 ** -43)]),
            (1024, 300, [(700, 2.0 ** -45 * 1.5), (701, 2.0 ** -72), (900, -2.0 ** -60)])):
        x = np.zeros(n, np.float32)
        x[: 2 * pairs] = np.tile([1.0, -1.0], pairs)
        for at, v in put:
            x[at] = v
        rows.append(x)
    x = np.zeros(1024, np.float32)  # partial sums past 2^53 lowest bits by the small samples alone
    x[[0, 4, 8, 12]] = 1.0, 1.0, 1.0, 0.9375
    x[[20, 600]] = 2.0 ** -51
    x[32:512] = 2.0 ** -12 - 2.0 ** -26
    rows.append(x)
    return rows


@pytest.mark.parametrize("k", range(5))
@pytest.mark.parametrize("axis", ["channels", "spectra"])
def test_clip_of_cancelling_samples(lib, orc, cuda, k, axis):
    import mdsm_gb300 as m
    r = _rows()[k]
    x = np.tile(r, (3, 1)) if axis == "channels" else np.tile(r[:, None], (1, 16))
    x = np.ascontiguousarray(x)
    kc, ks = (0.5, 0.0) if axis == "channels" else (0.0, 0.5)  # (most samples become the mean)
    want = orc.rfi_clip(x.copy(), x.shape[1], kc, ks)
    d = cuda.from_numpy(x).cuda()
    m.rfi_clip_device(d, x.shape[0], x.shape[1], x.shape[1], kc, ks, dtype="f32")
    got = d.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("k", range(5))
def test_block_statistics_of_cancelling_samples(lib, orc, cuda, k):
    import mdsm_gb300 as m
    r = _rows()[k]
    y = np.zeros((2, 16384), np.float32)
    y[0, : r.size] = r
    y[1, 100: 100 + r.size] = r[::-1]
    cands, mean, rms, n = m.ref_detect_device(cuda.from_numpy(y).cuda(), 2.0, 0.5, 1e9)
    with np.errstate(all="ignore"):
        _, om, orms = orc.ref_detect(y, 2.0, 0.5, 1e9)
    assert np.array_equal([mean, rms], [om, orms], equal_nan=True)
