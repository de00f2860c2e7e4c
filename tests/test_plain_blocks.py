"""CTA sizes of the plain engine: kernels of many registers run CTAs of one
warp unless the caller names a size; every size gives the oracle's bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257])
@pytest.mark.parametrize("mode,opts,cta", [("plain", {}, 32), ("plain", dict(block_size=256), 256),
                                           ("plain", dict(block_size=100), 32),
                                           ("regroup", dict(plain_below=1 << 40, block_size=512), 32)])
def test_large_kernel(n, mode, opts, cta):
    from loom_b200 import api
    from loom_b200 import scenes as S
    from oracle import oracle as O

    table, _ = S.pack([S.cornell_request(16, 16, 2, seed=9)])
    want = O.Interp("sphere_pt_f32").run([np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32)], table=table)
    with api.Function("sphere_pt_f32", n, mode, **opts) as f:
        got = f.launch_host([api.Broadcast(0, "u32"), api.Iota()], n, table=table)
        s = f.stats(raise_on_device_error=True)
    assert s["grid"] == -(-n // cta)
    for g, w in zip(got, want):
        assert np.array_equal(g.view(np.uint32), np.asarray(w).view(np.uint32))


@pytest.mark.parametrize("opts,cta", [({}, 256), (dict(block_size=64), 64)])
def test_small_kernel(opts, cta):
    from loom_b200 import api
    from oracle import oracle as O

    x = np.arange(1, 1001, dtype=np.uint64)
    (want,) = O.Interp("collatz_u64").run([x])
    with api.Function("collatz_u64", 1000, "plain", **opts) as f:
        assert np.array_equal(f(x), want)
        assert f.stats()["grid"] == -(-1000 // cta)
