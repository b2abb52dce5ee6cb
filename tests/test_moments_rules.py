"""A launch that folds the rows' moments into its store (served blocks) cannot cut the channels into parts, so
a plan whose kernel was chosen for its parts runs the packed kernel there; a plan whose tiles fill the SMs
runs the same kernel with and without moments."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def kernels(lib, tmp_path_factory):
    from mdsm_gb300 import build
    from mdsm_gb300._lib import DTYPES
    exe = str(tmp_path_factory.mktemp("rules") / "moments_rules")
    objs = [os.path.join(build.BUILD, f) for f in sorted(os.listdir(build.BUILD))
            if f.endswith(".o")]
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    subprocess.run([build.nvcc(), "-std=c++17", *build.ARCH, "-I", build.CSRC, "-I",
                    os.path.join(ROOT, "include"), "-cudart", "shared", "-Xlinker",
                    "-rpath," + os.path.join(cuda, "lib64"),
                    os.path.join(ROOT, "tests", "drivers", "moments_rules.cpp"), *objs, "-o", exe,
                    "-lpthread"], check=True, capture_output=True)

    def f(dtype, *args):
        w = subprocess.run([exe, str(DTYPES[dtype]), *map(str, args)], check=True,
                           capture_output=True, text=True).stdout.split()
        assert w[0::2] == ["sums", "moments"]
        return w[1], w[3]
    return f


@pytest.mark.parametrize("dtype,nchans,nsamp,ndms,step,want", [
    ("u8", 1734, 3852, 575, 0.5, ("gs", "packed")),     # short: a few tiles, cut into parts
    ("u8", 106, 2896, 116, 0.3, ("gs", "packed")),
    ("u8", 4096, 65536, 4096, 0.244140625, ("gs", "gs")),  # many tiles: one part either way
    ("u8", 801, 20000, 300, 0.23, ("gs", "gs"))])
def test_kernel_with_and_without_moments(kernels, dtype, nchans, nsamp, ndms, step, want):
    assert kernels(dtype, nchans, nsamp, ndms, step) == want
