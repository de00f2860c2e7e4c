"""Plain launches at every CTA size that the options take: sizes that a
kernel's registers do not allow run as the largest that they do, profiled or
not, and give the bits of the default size (whose parity with the golden
fixtures the engines' tests check)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [False, True])
@pytest.mark.parametrize("block", [256, 288, 640, 768, 832, 1024])
@pytest.mark.parametrize("kernel", ["pt_const_40", "pt2_const_40", "primary_const_256", "sphere_pt_f32", "threefry_u32"])
def test_named_sizes(golden, golden_extra, kernel, block, profile):
    from loom_b200 import api

    ins, _ = golden(kernel)
    n = min(len(ins[0]), 2048)
    with api.Function(kernel, n, "plain", block_size=256) as f:
        want = f.launch_host([a[:n] for a in ins], n, table=golden_extra(kernel).get("table"))
    with api.Function(kernel, n, "plain", block_size=block, profile=profile) as f:
        got = f.launch_host([a[:n] for a in ins], n, table=golden_extra(kernel).get("table"))
        s = f.stats(raise_on_device_error=True)
    assert np.asarray(got).tobytes() == np.asarray(want).tobytes()
    assert s["threads"] == n and s["grid"] >= -(-n // block)
    if block == 256:
        assert s["grid"] == -(-n // 256)
