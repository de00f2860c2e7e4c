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


@pytest.mark.parametrize("mode,opts", [("plain", {}), ("plain", dict(block_size=64)), ("regroup", dict(plain_below=1 << 40))])
@pytest.mark.parametrize("kernel,n", [("sphere_pt_f32", 33), ("sphere_pt_f32", 768), ("sphere_pt_f32", 2048), ("pt_const_40", 700), ("threefry_u32", 2048)])
def test_profiled_launches_run_what_they_describe(golden, golden_extra, kernel, n, mode, opts):
    """The grid of a profiled launch is that of the launch without counters,
    part-filled warps included, and its lane efficiency speaks of them."""
    from loom_b200 import api

    ins, _ = golden(kernel)
    n = min(n, len(ins[0]))
    got = {}
    for profile in (False, True):
        with api.Function(kernel, n, mode, profile=profile, **opts) as f:
            out = f.launch_host([a[:n] for a in ins], n, table=golden_extra(kernel).get("table"))
            s = f.stats(raise_on_device_error=True)
        got[profile] = np.asarray(out).tobytes(), s["grid"], s["lane_efficiency"]
    assert got[False][:2] == got[True][:2]
    per_warp = n / got[True][1] if got[True][1] > -(-n // 32) else 32
    assert 0 < got[True][2] <= min(32.0, np.ceil(per_warp)) / 32 + 1e-9
