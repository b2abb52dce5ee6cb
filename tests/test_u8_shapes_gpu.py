"""The uint8 brute-force tile shapes (38, 32 and 16 trials; 512 and 768 samples), each where the plan's
size or span of shifts chooses it, whole or with the channels cut into parts that add up, with
partial tiles, blocks and channel chunks, and on a buffer that ends with the last sample the plan
needs.  Exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


SEEN = set()
PLANS = [(64, 200, 5, 0.5), (33, 1500, 76, 0.5), (40, 4097, 130, 0.3), (16, 9000, 400, 0.3),
         (17, 40000, 600, 0.2), (512, 6000, 40, 1.5), (1024, 20000, 70, 1.5), (600, 20011, 97, 2.2),
         (48, 30011, 1000, 0.4), (9, 4, 1, 0.5), (32, 70001, 1140, 0.1), (700, 9001, 380, 1.4)]


@pytest.mark.parametrize("nchans,nsamp,ndms,dmstep", PLANS)
@pytest.mark.parametrize("out_dtype", ["i32", "f32"])
def test_u8_tile_shapes(lib, orc, cuda, nchans, nsamp, ndms, dmstep, out_dtype):
    import mdsm_gb300 as m
    plan = m.BrutePlan(nchans, 1500.0, -300.0 / nchans, 64e-6, nsamp, [(3.0, dmstep, ndms)],
                       in_dtype="u8", out_dtype=out_dtype)
    i = plan.info
    assert i.kernel == 2
    SEEN.add((i.dm_block, i.time_tile))
    stride = i.in_stride
    n = (nchans - 1) * stride + (nsamp + i.maxshift + 15) // 16 * 16
    flat = np.random.default_rng(nchans + ndms).integers(0, 256, n, dtype=np.uint8)
    d_in = cuda.from_numpy(flat).cuda()
    d_out = cuda.zeros((ndms, nsamp + 3), device="cuda",
                       dtype=cuda.int32 if out_dtype == "i32" else cuda.float32)
    plan.dedisperse_device(d_in, d_out)
    got = d_out.cpu().numpy()
    x = np.zeros(nchans * stride, np.uint8)
    x[:n] = flat
    want = orc.dedisperse(x.reshape(nchans, stride), plan.shift_table(), nsamp)
    assert np.array_equal(got[:, :nsamp], want.astype(got.dtype))
    assert not got[:, nsamp:].any()
    plan.check()


@pytest.mark.parametrize("dtype", ["u16", "i16"])
@pytest.mark.parametrize("out_dtype", ["i32", "f32"])
@pytest.mark.parametrize("nchans,nsamp,ndms", [(250, 900, 20), (641, 2500, 35), (33, 700, 5)])
def test_16_bit_parts(lib, orc, cuda, dtype, out_dtype, nchans, nsamp, ndms):
    """Calls with few tiles of 16-bit samples: the channels cut into parts (float output only
    where whole numbers stay within 2^24), with samples at the ends of their range."""
    import mdsm_gb300 as m
    plan = m.BrutePlan(nchans, 1500.0, -300.0 / nchans, 64e-6, nsamp, [(0.0, 0.4, ndms)],
                       in_dtype=dtype, out_dtype=out_dtype)
    assert plan.info.kernel == 3
    info = np.iinfo(np.uint16 if dtype == "u16" else np.int16)
    x = np.random.default_rng(nchans).integers(info.min, info.max + 1, plan.input_shape()).astype(
        info.dtype)
    x[::3] = info.max
    x[1::5] = info.min
    d_in = plan.alloc_input()
    d_in[: x.size].copy_(cuda.from_numpy(x).reshape(-1))
    d_out = plan.alloc_output()
    plan.dedisperse_device(d_in, d_out)
    want = orc.dedisperse(x, plan.shift_table(), nsamp)
    assert np.array_equal(d_out.cpu().numpy(), want.astype(d_out.cpu().numpy().dtype))


def test_every_shape_ran(lib, cuda):
    if len(SEEN) > 3:  # (the whole file ran)
        assert {38, 32, 16} <= {s[0] for s in SEEN} and {512, 768} <= {s[1] for s in SEEN}, SEEN
