"""What a plan says about itself where the group sums run it though the packed staging does not fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_group_sums_without_packed_staging(lib, orc, cuda):
    import mdsm_gb300 as m
    plan = m.BrutePlan(1024, 1500.0, -300.0 / 1024, 64e-6, 100000, [(0.0, 4.0, 38)], in_dtype="u8",
                       out_dtype="i32")
    st = plan.stage_info(0)
    assert st.kernel == 5 and plan.info.kernel == 2 and plan.info.dm_block == st.dm_block
    x = np.random.default_rng(2).integers(0, 256, plan.input_shape()).astype(np.uint8)
    d_in = plan.alloc_input()
    d_in[: x.size].copy_(cuda.from_numpy(x).reshape(-1))
    d_out = plan.alloc_output()
    plan.dedisperse_device(d_in, d_out)
    plan.check()
    want = orc.dedisperse(x, plan.shift_table(), 100000)
    assert np.array_equal(d_out.cpu().numpy(), want)
