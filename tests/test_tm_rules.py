"""The rules by which a float stage takes the tensor-memory kernel, compiled for the host.

The tensor-memory kernel shares out the registers that it is launched with; a build in which it does not
come out at exactly these is not used, and its stages keep the generic kernel (no call fails for it).

Its allocation of an SM's tensor memory would wait, without a bound, for another kernel's CTA that holds some
there, so it asks for so much shared memory that it shares its SMs with no other CTA."""
import os
import platform
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mdsm_gb300", "csrc")


@pytest.fixture(scope="module")
def rules(lib, tmp_path_factory):
    from mdsm_gb300 import build
    exe = str(tmp_path_factory.mktemp("rules") / "tm_rules")
    objs = [os.path.join(build.BUILD, f) for f in sorted(os.listdir(build.BUILD))
            if f.endswith(".o") and f != "tmsum.cu.o"]
    assert platform.machine() in build.BUILD and objs
    subprocess.run([build.nvcc(), "-std=c++17", *build.ARCH, "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), "--expt-relaxed-constexpr",
                    os.path.join(ROOT, "tests", "drivers", "tm_rules.cu"), *objs, "-o", exe,
                    "-lpthread"], check=True, capture_output=True)

    def f(*args):
        r = subprocess.run([exe, *map(str, args)], check=True, capture_output=True, text=True)
        return tuple(map(int, r.stdout.split()))
    return f


REGS = int(re.search(r"kTmRegs = (\d+)", open(os.path.join(CSRC, "tmsum.cu")).read()).group(1))
SMEM_PER_SM = 228 * 1024  # bytes of shared memory per SM (sm_100 family)
SMEM_PER_CTA_RESERVED = 1024


def test_other_register_counts_keep_the_generic_kernel(rules):
    assert rules(REGS)[0] >= 0
    for other in (0, REGS - 8, REGS + 8):
        assert rules(other)[0] == -1


@pytest.mark.parametrize("ndms,nsamp", [(496, 32000), (96, 200000), (2000, 9000)])
def test_no_other_cta_on_its_sms(rules, ndms, nsamp):
    shape, smem = rules(REGS, ndms, nsamp)
    assert shape >= 0
    left = SMEM_PER_SM - (smem + SMEM_PER_CTA_RESERVED)
    assert 0 <= left < SMEM_PER_CTA_RESERVED
