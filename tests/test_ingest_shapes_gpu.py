"""Unpacking and time downsampling over the shapes where their kernels change: channel tiles and
their remainders, counts that are not multiples of 4, aligned and unaligned outputs, partial last
tiles; float sums of samples whose exponents lie far apart.  Bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TORCH = {"u8": "uint8", "u16": "uint16", "i16": "int16", "i32": "int32", "f32": "float32"}


@pytest.mark.parametrize("nbits,dtype", [(1, "u8"), (2, "f32"), (4, "u16"), (8, "u8"), (8, "f32"),
                                         (16, "u16"), (16, "i16"), (16, "f32"), (32, "f32")])
@pytest.mark.parametrize("nchans,nspec,stride,col0", [(8, 1, 16, 0), (128, 128, 128, 0),
                                                      (136, 129, 160, 16), (264, 401, 416, 3),
                                                      (40, 33, 37, 1), (24, 65, 80, 0)])
@pytest.mark.parametrize("shift", [0, 1])
def test_unpack_shapes(lib, orc, cuda, nbits, dtype, nchans, nspec, stride, col0, shift):
    from mdsm_gb300 import sigproc
    if nbits == 32 and shift:
        pytest.skip("float samples are aligned")
    rng = np.random.default_rng(nchans + nspec)
    if shift:
        nchans -= 8 if nbits < 8 else 1  # counts off a multiple of 4 take the general kernel
        if nchans == 0:
            pytest.skip("no channels")
    n = nchans * nspec
    raw = rng.integers(0, 256, n * nbits // 8, dtype=np.uint8)
    if nbits == 32:
        raw = rng.standard_normal(n).astype(np.float32).view(np.uint8)
    want = orc.unpack(raw, nbits).reshape(nspec, nchans).T
    if dtype == "i16":
        want = raw.view("<i2").reshape(nspec, nchans).T
    ncol = max(stride, col0 + nspec)
    out = cuda.zeros((nchans, ncol), dtype=getattr(cuda, TORCH[dtype]), device="cuda")
    sigproc.unpack_device(cuda.from_numpy(raw).cuda(), nspec, nchans, nbits, out, dtype, ncol, col0)
    got = out.cpu().numpy()
    assert np.array_equal(got[:, col0:col0 + nspec], want.astype(got.dtype))
    assert not got[:, :col0].any() and not got[:, col0 + nspec:].any()


@pytest.mark.parametrize("tin,tout", [("u8", "u16"), ("u8", "i32"), ("u16", "i32"), ("i16", "i32"),
                                      ("f32", "f32")])
@pytest.mark.parametrize("b", [2, 4, 8])
@pytest.mark.parametrize("length,stride,ostride", [(7, 16, 16), (4096, 4096, 2048),
                                                   (5003, 5008, 2512), (1001, 1003, 777)])
def test_downsample_shapes(lib, cuda, tin, tout, b, length, stride, ostride):
    from mdsm_gb300 import _lib
    rng = np.random.default_rng(length + b)
    nchans = 5
    if tin == "f32":
        x = rng.standard_normal((nchans, stride)).astype(np.float32)
        x[1] *= np.exp2(rng.integers(-70, 70, stride)).astype(np.float32)
        x[2, ::3] = 0.0
        x[3] = -0.0
        x[4, ::5] *= np.float32(1e-42)
    else:
        info = np.iinfo(np.dtype(TORCH[tin]))
        x = rng.integers(info.min, info.max + 1, (nchans, stride)).astype(TORCH[tin])
    nout = length // b
    d_in = cuda.from_numpy(x).cuda()
    d_out = cuda.zeros((nchans, ostride), dtype=getattr(cuda, TORCH[tout]), device="cuda")
    _lib.check(_lib.load().mdsm_downsample_device(
        ctypes.c_void_p(d_in.data_ptr()), _lib.DTYPES[tin], nchans, stride, length, b, 0,
        ctypes.c_void_p(d_out.data_ptr()), _lib.DTYPES[tout], ostride,
        ctypes.c_void_p(cuda.cuda.current_stream().cuda_stream)))
    got = d_out.cpu().numpy()
    acc = np.zeros((nchans, nout), np.float64 if tin == "f32" else np.int64)
    for k in range(b):
        acc = acc + x[:, k:nout * b:b].astype(acc.dtype)
    want = acc.astype(got.dtype)
    assert np.array_equal(got[:, :nout].view(np.uint8), want.view(np.uint8))
    assert not got[:, nout:].any()
