"""The tensor-memory kernel shares out the registers that it is launched with; a build in which it does not
come out at exactly these is not used, and its stages keep the generic kernel (no call fails for it)."""
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

    def f(regs):
        return int(subprocess.run([exe, str(regs)], check=True, capture_output=True, text=True).stdout)
    return f


def test_other_register_counts_keep_the_generic_kernel(rules):
    regs = int(re.search(r"kTmRegs = (\d+)", open(os.path.join(CSRC, "tmsum.cu")).read()).group(1))
    assert rules(regs) >= 0
    for other in (0, regs - 8, regs + 8):
        assert rules(other) == -1
