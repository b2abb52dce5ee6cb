"""Brute-force plans of 8- and 16-bit samples whose neighbouring channels share patterns of shifts (sums of
groups of channels): both blocks of trials (60, 38), whole or with the channels cut into parts, DM ranges
with steps, partial tiles, blocks and groups of channels, samples at the ends of their range, output that
is not on 8-byte boundaries, and a buffer no longer than the plan asks for.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GROUPS = 5  # mdsm_stage_info's kernel
SEEN = set()
PLANS = [  # type, nchans, nsamp, segments, bandwidth
    ("u8", 1203, 9000, [(0.0, 0.23, 181)], 100.0),
    ("u8", 1500, 15000, [(0.0, 0.2, 39)], 300.0),
    ("u8", 2050, 5000, [(0.0, 0.2, 61), (12.2, 0.4, 30), (24.2, 0.8, 31)], 300.0),
    ("u8", 801, 20000, [(0.0, 0.23, 300)], 100.0),
    ("u8", 1600, 30000, [(0.0, 0.2, 38)], 100.0),
    ("u8", 152, 6086, [(0.0, 0.85, 204), (173.4, 1.7, 102), (346.8, 3.4, 103)], 300.0),
    ("i16", 1313, 7000, [(0.0, 0.3, 61)], 100.0),
    ("i16", 600, 3542, [(0.0, 0.2, 300)], 300.0),
    ("u16", 1999, 2007, [(250.0, 0.26, 165)], 100.0),
    ("u16", 114, 3176, [(0.0, 0.33, 774), (255.0, 0.66, 387), (510.0, 1.32, 387)], 100.0),
]


@pytest.mark.parametrize("dtype,nchans,nsamp,segs,bw", PLANS)
@pytest.mark.parametrize("out_dtype", ["i32", "f32"])
def test_group_sums(lib, orc, cuda, dtype, nchans, nsamp, segs, bw, out_dtype):
    import mdsm_gb300 as m
    plan = m.BrutePlan(nchans, 1500.0, -bw / nchans, 64e-6, nsamp, segs, in_dtype=dtype,
                       out_dtype=out_dtype)
    i, st = plan.info, plan.stage_info(0)
    if out_dtype == "f32" and dtype != "u8" and st.kernel != GROUPS:
        pytest.skip("float parts would not be exact: whole tiles are too few, or summed in floats")
    assert st.kernel == GROUPS
    SEEN.add((dtype, i.dm_block))
    np_t = {"u8": np.uint8, "u16": np.uint16, "i16": np.int16}[dtype]
    lo, hi = np.iinfo(np_t).min, np.iinfo(np_t).max
    n = i.in_bytes // np.dtype(np_t).itemsize
    flat = np.random.default_rng(nchans).integers(lo, hi + 1, n).astype(np_t)
    for c in range(0, nchans - 1, 5):
        flat[c * i.in_stride:(c + 1) * i.in_stride] = hi if c % 2 else lo
    flat[2 * i.in_stride:10 * i.in_stride] = hi  # a whole group of channels
    d_in = cuda.from_numpy(flat).cuda()
    x = np.zeros(max(n, nchans * i.in_stride), np_t)
    x[:n] = flat
    want = orc.dedisperse(x[: nchans * i.in_stride].reshape(nchans, i.in_stride), plan.shift_table(),
                          nsamp)
    for pad in (0, 3):
        d_out = cuda.full((i.ndms, nsamp + pad), 7, device="cuda",
                          dtype=cuda.int32 if out_dtype == "i32" else cuda.float32)
        plan.dedisperse_device(d_in, d_out)
        got = d_out.cpu().numpy()
        assert np.array_equal(got[:, :nsamp], want.astype(got.dtype))
        assert (got[:, nsamp:] == 7).all()
    plan.check()


def test_both_blocks_ran(lib, cuda):
    if len(SEEN) > 3:  # (the whole file ran)
        assert {("u8", 60), ("u8", 38), ("i16", 60), ("i16", 38), ("u16", 60), ("u16", 38)} == SEEN


def test_group_sums_fold_moments(lib, orc, cuda):
    """A served beam: the rows' exact moments come from the sums' store."""
    import mdsm_gb300 as m
    from mdsm_gb300 import synth
    from mdsm_gb300.serving import Server
    nchans, nsamp, segs = 801, 20000, [(0.0, 0.23, 300)]
    plan = m.BrutePlan(nchans, 1500.0, -100.0 / nchans, 64e-6, nsamp, segs, out_dtype="i32")
    assert plan.stage_info(0).kernel == GROUPS
    srv = Server(max_inflight=1, nwidths=7, threshold=6.0, cand_cap=4096)
    b = srv.add_beam(nchans, 1500.0, -100.0 / nchans, 64e-6, nsamp, segs)
    x = synth.gaussian_u8(nchans, nsamp + srv.beam_info(b).maxshift, 5)
    synth.inject(x, 1500.0, -100.0 / nchans, 64e-6, [(7000, 30.0, 8, 30.0)], K=4148.741601)
    assert srv.submit(b, x) is not None
    (r,) = srv.results(1)
    srv.close()
    y = orc.dedisperse(x, plan.shift_table(), nsamp)
    dm, samp, wid, snr = orc.boxcar_detect(y, 7, 6.0)
    assert len(dm)
    assert np.array_equal(r["cands"]["dm_idx"], dm) and np.array_equal(r["cands"]["sample"], samp)
    assert np.array_equal(r["cands"]["width"], wid) and np.array_equal(r["cands"]["snr"], snr)
