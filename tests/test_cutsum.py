"""The exact float sums of the RFI clip's and the detector's statistics (mdsm_gb300/csrc/cutsum.cuh),
compiled for the host: where they say that they are exact, they equal the left-to-right double sum bit for
bit.  Ordinary data has to be summed exactly; data with remainders past the third cut, cancelling sums,
partial sums at the edge of 53 bits, infinities and NaN may only be declined."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def cut_sum(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("cutsum") / "cutsum.so")
    drivers = os.path.join(ROOT, "tests", "drivers")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(drivers, "cutsum_host.cpp"), "-I",
                    os.path.join(drivers, "host_cuda"), "-I",
                    os.path.join(ROOT, "mdsm_gb300", "csrc")], check=True)
    lib = ctypes.CDLL(so)

    def f(x, biggest=None):
        x = np.ascontiguousarray(x, np.float32)
        if biggest is None:  # as the clip picks it from a run's first 16 samples
            m = np.abs(x[:16]).reshape(4, 4).max(axis=1) if len(x) >= 32 else np.zeros(4, np.float32)
            biggest = max(min(m[0], m[1]), min(m[2], m[3]))
        s = ctypes.c_double()
        ok = lib.cut_sum(x.ctypes.data_as(ctypes.c_void_p), len(x), ctypes.c_float(biggest),
                         ctypes.byref(s))
        return bool(ok), s.value
    return f


def _chain(x):
    s = 0.0
    for v in np.asarray(x, np.float32).astype(np.float64):
        s = s + v
    return s


def _check(cut_sum, x, must=False):
    ok, got = cut_sum(x)
    assert ok or not must
    if ok:
        want = _chain(x)
        assert np.float64(got).tobytes() == np.float64(want).tobytes(), (got, want)
    return ok


def _remainders(n, pairs, *put):
    x = np.zeros(n, np.float32)
    x[: 2 * pairs] = np.tile([1.0, -1.0], pairs)
    for at, v in put:
        x[at] = v
    return x


REMAINDERS = [
    # a remainder below half the last place of those already seen, alone or after they cancelled
    _remainders(64, 32, (20, 2.0 ** -42), (21, -2.0 ** -42), (22, 0.0), (23, 0.0),
                (62, 2.0 ** -68), (63, 0.0)),
    _remainders(1024, 16, (40, 2.0 ** -43), (60, 2.0 ** -70)),
    _remainders(1024, 16, (40, 2.0 ** -43), (60, 2.0 ** -70), (70, -2.0 ** -43)),
    _remainders(1024, 16, (40, 2.0 ** -45 * 1.5), (41, 2.0 ** -72), (900, -2.0 ** -60)),
]


@pytest.mark.parametrize("k", range(len(REMAINDERS)))
def test_small_remainders_are_not_dropped(cut_sum, k):
    _check(cut_sum, REMAINDERS[k])


def test_partial_sums_beyond_53_bits_are_declined(cut_sum):
    """The first third's sum stays below 2^53 lowest bits, the sum of the second takes it past them:
    the chain loses a lowest bit at 4.0 and another after it."""
    x = np.zeros(1024, np.float32)
    x[[0, 4, 8, 12]] = 1.0, 1.0, 1.0, 0.9375
    x[20] = 2.0 ** -51
    x[32:512] = 2.0 ** -12 - 2.0 ** -26
    x[600] = 2.0 ** -51
    _check(cut_sum, x)


def test_cancelling_samples_of_many_sizes(cut_sum):
    rng = np.random.default_rng(3)
    for k in range(300):
        n = int(rng.integers(32, 1025))
        x = np.ldexp(rng.choice([-1.0, 1.0], n) * (1 + rng.integers(0, 1 << 10, n) / 1024.0),
                     -rng.integers(0, 81, n)).astype(np.float32)
        big = rng.permutation(n)[: n // 4 * 2]
        x[big[::2]] = x[big[1::2]] = 0
        x[big[::2]] = np.float32(1.0) * rng.integers(1, 5, len(big) // 2)
        x[big[1::2]] = -x[big[::2]]
        if k % 2:
            x[np.abs(x) > 2.0 ** -40] = 0
            x[:16] = np.tile([1.0, -1.0], 8)
        _check(cut_sum, x)


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (3.0, 1.0), (1e-6, 0.0), (16.0, 128.0),
                                          (1000.0, 0.0)])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 500, 1023, 1024])
def test_ordinary_samples_are_summed(cut_sum, scale, offset, n):
    x = np.random.default_rng(n).standard_normal(n, dtype=np.float32) * np.float32(scale)
    _check(cut_sum, x + np.float32(offset), must=n >= 32)


def test_samples_that_are_not_finite_are_declined(cut_sum):
    x = np.random.default_rng(1).standard_normal(200, dtype=np.float32)
    for at in (0, 40, 199):
        for v in (np.inf, -np.inf, np.nan):
            y = x.copy()
            y[at] = v
            assert not cut_sum(y)[0]
    y = x.copy()
    y[50], y[60] = np.inf, -np.inf
    assert not cut_sum(y)[0]
