"""Float samples with int32 output: the float sums truncated to int32 (infinite and too large sums to
the type's ends, NaN to 0), at sizes where float output takes the tensor-memory kernel and where it takes
the generic one, in brute-force plans and in both stages of subband plans (float samples, and 8-bit
samples summed in floats)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _trunc(y):
    """int32 of a float as the device converts it."""
    with np.errstate(invalid="ignore"):
        z = np.clip(np.trunc(y.astype(np.float64)), -2.0 ** 31, 2.0 ** 31 - 1)
    return np.where(np.isnan(y), 0, z).astype(np.int64).astype(np.int32)


@pytest.mark.parametrize("nchans,nsamp,ndms,tm", [(257, 1536 * 40 + 1, 100, True),
                                                  (300, 6228, 403, True), (33, 1500, 20, False)])
def test_float_brute_i32(lib, cuda, nchans, nsamp, ndms, tm):
    import mdsm_gb300 as m
    args = (nchans, 1500.0, -100.0 / nchans, 64e-6, nsamp, [(0.0, 0.2, ndms)])
    kw = dict(in_dtype="f32", shift_mode="fp64_round")
    ints = m.BrutePlan(*args, out_dtype="i32", **kw)
    generic = m.BrutePlan(*args, out_dtype="i32", kernel=1, **kw)
    floats = m.BrutePlan(*args, out_dtype="f32", **kw)
    assert (floats.info.kernel == 4) == tm
    d_in = floats.alloc_input()
    g = cuda.Generator(device="cuda").manual_seed(nchans)
    d_in.copy_(cuda.randn(d_in.shape, generator=g, device="cuda") * 37.0)
    d_in[5::4001] = float("inf")
    d_in[9::5003] = float("nan")
    d_in[11::3001] = -3e9
    outs = []
    for p in (ints, generic, floats):
        d_out = p.alloc_output()
        p.dedisperse_device(d_in, d_out)
        p.check()
        outs.append(d_out.cpu().numpy())
    want = _trunc(outs[2])
    assert len(np.unique(want)) > 100
    assert np.array_equal(outs[1], want)
    assert np.array_equal(outs[0], want)


@pytest.mark.parametrize("in_dtype,acc", [("f32", "auto"), ("u8", "f32")])
@pytest.mark.parametrize("nsamp,ncalls,calldms,dmstep", [(12000, 32, 24, 0.1), (9004, 40, 32, 0.25)])
def test_float_subband_i32(lib, cuda, in_dtype, acc, nsamp, ncalls, calldms, dmstep):
    import mdsm_gb300 as m
    nchans, nsubs = 1024, 64
    p = dict(lowdm=0.0, highdm=ncalls * calldms * dmstep, dmstep=dmstep,
             sub_dmstep=calldms * dmstep, ncalls=ncalls, calldms=calldms)
    outs = []
    for out_dtype in ("i32", "f32"):
        plan = m.SubbandPlan(nchans, 1500.0, -300.0 / nchans, 64e-6, nsamp, nsubs, [p],
                             in_dtype=in_dtype, out_dtype=out_dtype, acc=acc)
        d_in = plan.alloc_input()
        g = cuda.Generator(device="cuda").manual_seed(nsamp)
        if in_dtype == "f32":
            d_in.copy_(cuda.randn(d_in.shape, generator=g, device="cuda") * 37.0)
        else:
            d_in.copy_(cuda.randint(0, 256, d_in.shape, generator=g, device="cuda"))
        d_out = plan.alloc_output()
        plan.dedisperse_device(d_in, d_out)
        plan.check()
        outs.append(d_out.cpu().numpy())
    want = _trunc(outs[1])
    assert len(np.unique(want)) > 100
    assert np.array_equal(outs[0], want)
