"""Float shift-and-sums through tensor memory, in brute-force plans and both subband stages: every
block of trials (16, 12, 8), partial tiles of 1536 samples and segments of 12, partial DM blocks, odd
channel counts, spans from none to the widest that are taken, infinities, NaN and -0, and a buffer
no longer than the plan asks for.  The sums run channel by channel in 32-bit floats, so
they are compared bit for bit with the same sums in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEEN = set()
PLANS = [  # nchans, nsamp, segments, bandwidth
    (257, 1536 * 40 + 1, [(0.0, 0.2, 100)], 100.0),
    (128, 1536 * 21 - 1, [(0.0, 0.2, 497)], 100.0),
    (92, 61418, [(0.0, 0.2, 24), (4.8, 0.4, 12), (9.6, 0.8, 11)], 100.0),
    (851, 8429, [(0.0, 0.2, 121)], 100.0),
    (300, 1536 * 4 + 12 * 7, [(0.0, 0.3, 403)], 100.0),
    (512, 30011, [(0.0, 0.9, 65)], 100.0),
    (699, 9391, [(9.2, 0.46, 583)], 100.0),
    (64, 120000, [(0.0, 0.0, 96)], 100.0),
    (1024, 9000, [(397.0, 0.25, 320)], 100.0),
    (600, 14000, [(0.0, 0.2, 333)], 300.0),
]


def _sum(x, shifts, n):
    out = np.zeros((shifts.shape[0], n), np.float32)
    for d in range(shifts.shape[0]):
        for c in range(shifts.shape[1]):
            out[d] += x[c, shifts[d, c]:shifts[d, c] + n]
    return out


def _same(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])


@pytest.mark.parametrize("nchans,nsamp,segs,bw", PLANS)
def test_float_brute(lib, cuda, nchans, nsamp, segs, bw):
    import mdsm_gb300 as m
    plan = m.BrutePlan(nchans, 1500.0, -bw / nchans, 64e-6, nsamp, segs, in_dtype="f32",
                       out_dtype="f32", shift_mode="fp64_round")
    i = plan.info
    assert i.kernel == 4 and i.time_tile == 1536
    SEEN.add(i.dm_block)
    rng = np.random.default_rng(nchans)
    n = i.in_bytes // 4
    flat = rng.standard_normal(n, dtype=np.float32)
    flat[rng.integers(0, n, 40)] = np.inf
    flat[rng.integers(0, n, 40)] = -np.inf
    flat[rng.integers(0, n, 40)] = np.nan
    d_in = cuda.from_numpy(flat).cuda()
    x = np.zeros(max(n, nchans * i.in_stride), np.float32)
    x[:n] = flat
    x = x[: nchans * i.in_stride]
    want = _sum(x.reshape(nchans, i.in_stride), plan.shift_table(), nsamp)
    for pad in (0, 3):  # rows that do and do not start on 16-byte boundaries
        d_out = cuda.full((i.ndms, nsamp + pad), 7.0, device="cuda")
        plan.dedisperse_device(d_in, d_out)
        got = d_out.cpu().numpy()
        _same(np.ascontiguousarray(got[:, :nsamp]), want)
        assert (got[:, nsamp:] == 7.0).all()
    zeros = cuda.full((n,), -0.0, device="cuda")
    plan.dedisperse_device(zeros, d_out)
    assert not np.signbit(d_out.cpu().numpy()[:, :nsamp]).any()  # the sum starts from +0
    plan.check()


def test_every_block_was_run(lib, cuda):
    assert SEEN == {16, 12, 8}, SEEN


def test_asked_for_kernels(lib, cuda):
    """A call that names the generic kernel, or its block, gets it."""
    import mdsm_gb300 as m
    for kw in (dict(kernel=1), dict(dm_block=16), dict(dm_block=8)):
        p = m.BrutePlan(128, 1500.0, -100.0 / 128, 64e-6, 32000, [(0.0, 0.2, 497)], in_dtype="f32",
                        **kw)
        assert p.info.kernel == 1 and p.info.dm_block == kw.get("dm_block", 32)


@pytest.mark.parametrize("nsubs,nsamp,ncalls,calldms,dmstep,stage", [(64, 12000, 32, 24, 0.1, 1),
                                                                     (64, 9004, 40, 32, 0.25, 0)])
def test_float_subband(lib, cuda, nsubs, nsamp, ncalls, calldms, dmstep, stage):
    import mdsm_gb300 as m
    nchans = 1024
    p = dict(lowdm=0.0, highdm=ncalls * calldms * dmstep, dmstep=dmstep,
             sub_dmstep=calldms * dmstep, ncalls=ncalls, calldms=calldms)
    plan = m.SubbandPlan(nchans, 1500.0, -300.0 / nchans, 64e-6, nsamp, nsubs, [p], in_dtype="f32")
    assert plan.stage_info(stage).kernel == 4
    i = plan.info
    x = np.random.default_rng(nsubs).standard_normal(plan.input_shape(), dtype=np.float32)
    d_in = plan.alloc_input()
    d_in[: x.size].copy_(cuda.from_numpy(x).reshape(-1))
    d_out = plan.alloc_output()
    plan.dedisperse_device(d_in, d_out)
    got = d_out.cpu().numpy().reshape(i.ndms, nsamp)
    s1, s2 = plan.stage_tables()
    n1, cps = nsamp + int(s2.max()), nchans // nsubs
    for j in range(ncalls):
        z = np.stack([_sum(x[b * cps:(b + 1) * cps], s1[j:j + 1, b * cps:(b + 1) * cps], n1)[0]
                      for b in range(nsubs)])
        rows = slice(j * calldms, (j + 1) * calldms)
        _same(got[rows], _sum(z, s2[rows], nsamp))
    plan.check()
