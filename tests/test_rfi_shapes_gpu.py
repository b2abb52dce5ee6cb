"""The RFI clip over the shapes where its kernels change: vector heads and tails, rows off
16-byte boundaries, runs of 1024 and their remainders, channel batches of a CTA and of a cluster,
constant rows, and rows whose statistics are infinite or not numbers.  Bit for bit against the
oracle (the statistics are exact or in a fixed order, so no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NP = {"u8": np.uint8, "i16": np.int16, "u16": np.uint16, "f32": np.float32}


def _block(dtype, nchans, stride, seed):
    rng = np.random.default_rng(seed)
    if dtype == "f32":
        x = rng.standard_normal((nchans, stride), dtype=np.float32) * 3 + 1
        x[:, ::37] += 60
    else:
        mean, sig = {"u8": (128, 16), "i16": (-50, 1000), "u16": (20000, 1500)}[dtype]
        x = rng.normal(mean, sig, (nchans, stride))
        x[:, ::37] += 40 * sig
        info = np.iinfo(NP[dtype])
        x = np.clip(np.rint(x), info.min, info.max).astype(NP[dtype])
    x[nchans // 2] = x[nchans // 2, 0]  # sigma 0
    if nchans > 8:
        x[3, ::2] = np.iinfo(NP[dtype]).max if dtype != "f32" else np.float32(3e38)
        x[3, 1::2] = np.iinfo(NP[dtype]).min if dtype != "f32" else np.float32(-3e38)
    return x


def _clip(torch, x, length, kc, ks, dtype, offset=0):
    import mdsm_gb300 as m
    flat = torch.zeros(x.size + offset, dtype=getattr(torch, np.dtype(NP[dtype]).name),
                       device="cuda")
    d = flat[offset:]
    d.copy_(torch.from_numpy(x).reshape(-1))
    m.rfi_clip_device(d, x.shape[0], x.shape[1], length, kc, ks, dtype=dtype)
    return d.cpu().numpy().reshape(x.shape)


@pytest.mark.parametrize("dtype", ["u8", "i16", "f32"])
@pytest.mark.parametrize("nchans,length,stride,offset", [
    (1, 1, 16, 0), (2, 5, 16, 0), (9, 1023, 1024, 0), (17, 1025, 1040, 0), (40, 2047, 2051, 0),
    (64, 999, 1008, 3), (511, 130, 144, 0), (513, 65, 80, 0), (1025, 47, 48, 0),
    (2049, 33, 48, 0), (4096, 31, 32, 0), (9000, 17, 32, 0), (16385, 16, 16, 0),
    (3, 40001, 40016, 0)])
def test_clip_shapes_match_oracle(lib, orc, cuda, dtype, nchans, length, stride, offset):
    x = _block(dtype, nchans, stride, nchans + length)
    for kc, ks in ((4.0, 4.0), (3.0, 0.0), (0.0, 2.5)):
        want = orc.rfi_clip(x.copy(), length, kc, ks)
        got = _clip(cuda, x, length, kc, ks, dtype, offset)
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8)), (kc, ks)


def test_clip_float_rows_without_finite_statistics(lib, orc, cuda):
    """Infinities and NaN among the samples: the same comparisons as in double."""
    x = _block("f32", 12, 2048, 5)
    x[0, 7] = np.inf
    x[1, 9] = -np.inf
    x[2, 11] = np.nan
    x[4, :2] = np.inf, -np.inf
    x[5, 5] = np.float32(1e-42)
    x[6] = 0.0
    x[6, 1::2] = -0.0
    for kc, ks in ((4.0, 0.0), (4.0, 4.0), (np.inf, 0.0)):
        want = orc.rfi_clip(x.copy(), 2000, kc, ks)
        got = _clip(cuda, x, 2000, kc, ks, "f32")
        assert np.array_equal(np.isnan(got), np.isnan(want)), (kc, ks)
        ok = ~np.isnan(want)
        assert np.array_equal(got[ok], want[ok]), (kc, ks)
