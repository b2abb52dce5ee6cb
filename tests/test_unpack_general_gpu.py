"""Unpacking off the tiles of 4-channel groups, for every sample width: channel counts off a multiple of 4
and raw data that does not start on a group of 4 samples, bit for bit; spectra that are not whole bytes (the
only such counts of 1- and 2-bit samples, and the odd ones of 4-bit samples) are refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbits,dtype", [(1, "u8"), (1, "f32"), (2, "u8"), (4, "u8"), (4, "f32"),
                                         (8, "u8"), (16, "u16"), (16, "i16"), (32, "f32")])
@pytest.mark.parametrize("nchans,nspec,offset,invert", [
    (12, 40, 0, 0), (4, 64, 0, 1), (133, 72, 0, 0), (34, 800, 0, 1), (1, 96, 0, 0), (33, 64, 1, 1),
    (128, 130, 1, 0), (96, 33, 1, 1), (264, 257, 1, 0), (128, 67, 0.5, 0), (133, 72, 0.5, 1)])
def test_unpack_general(lib, orc, cuda, nbits, dtype, nchans, nspec, offset, invert):
    from mdsm_gb300 import sigproc
    rng = np.random.default_rng(nchans + nspec + nbits)
    n = nchans * nspec
    raw = rng.integers(0, 256, n * nbits // 8, dtype=np.uint8)
    if nbits == 32:
        raw = rng.standard_normal(n).astype(np.float32).view(np.uint8)
    want = orc.unpack(raw, nbits).reshape(nspec, nchans).T
    if dtype == "i16":
        want = raw.view("<i2").reshape(nspec, nchans).T
    if invert:
        want = want[::-1]
    # a sample (below 8 bits: a byte of them), or one byte
    skip = 1 if offset == 0.5 else offset * max(1, nbits // 8)
    d_raw = cuda.zeros(raw.size + skip, dtype=cuda.uint8, device="cuda")
    d_raw[skip:].copy_(cuda.from_numpy(raw))
    stride, col0 = nspec + 9, 5
    td = {"u8": cuda.uint8, "u16": cuda.uint16, "i16": cuda.int16, "f32": cuda.float32}[dtype]
    out = cuda.zeros((nchans, stride), dtype=td, device="cuda")
    args = (d_raw[skip:], nspec, nchans, nbits, out, dtype, stride, col0, bool(invert))
    if nchans * nbits % 8:
        from mdsm_gb300 import MdsmError
        with pytest.raises(MdsmError):
            sigproc.unpack_device(*args)
        return
    sigproc.unpack_device(*args)
    got = out.cpu().numpy()
    assert np.array_equal(got[:, col0:col0 + nspec], want.astype(got.dtype))
    assert not got[:, :col0].any() and not got[:, col0 + nspec:].any()
