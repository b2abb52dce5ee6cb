"""The autotuner's file: a choice counts only for plans that run the same kernels, so a line written
when the plans had others (whose key named the sizes, the packed kernel and its span alone) is not used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _span(S, db):
    return max(int((S[i:i + db].max(axis=0) - S[i:i + db].min(axis=0)).max())
               for i in range(0, len(S), db))


def test_lines_for_other_kernels_are_not_used(lib, cuda, tmp_path, monkeypatch):
    import mdsm_gb300 as m
    from mdsm_gb300.batch import Batch
    nchans, nsamp, ndms = 801, 20000, 300
    plan = m.BrutePlan(nchans, 1500.0, -100.0 / nchans, 64e-6, nsamp, [(0.0, 0.23, ndms)],
                       out_dtype="i32")
    assert plan.stage_info(0).kernel == 5
    S = plan.shift_table()
    path = tmp_path / "tune"
    sizes = "%dx%dx%dk2" % (nchans, ndms, nsamp)
    path.write_text("".join("%ss%d; 1\n" % (sizes, _span(S, db)) for db in (16, 32, 38)))
    monkeypatch.setenv("MDSM_AUTOTUNE_CACHE", str(path))
    d_in, d_out = plan.alloc_input(), plan.alloc_output()
    b = Batch([plan])
    b.set_buffers([d_in], [d_out])
    choice = b.autotune()
    assert len(b.tune_times()) > 1  # the candidates were timed
    lines = path.read_text().splitlines()
    assert len(lines) == 4 and lines[-1].endswith(" %d" % choice)
    # and the new line is used
    c = Batch([plan])
    c.set_buffers([d_in], [d_out])
    assert c.autotune() == choice and not c.tune_times()
    b.close()
    c.close()
    assert np.isin(choice, range(32))
