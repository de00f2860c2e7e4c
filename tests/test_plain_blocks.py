"""CTA sizes of the plain engine: kernels of many registers run CTAs of one
warp unless the caller names a size, and small launches fewer threads than
lanes per warp, as the megakernel's do; every size gives the oracle's bits."""

import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _scene(n, seed=9):
    from loom_b200 import scenes as S
    from oracle import oracle as O

    table, _ = S.pack([S.cornell_request(16, 16, 2, seed=seed)])
    want = O.Interp("sphere_pt_f32").run([np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32)], table=table)
    return table, want


def _lanes(n):
    """Threads per warp of a small launch: the fewest, in powers of two,
    that 16 warps per SM hold."""
    import torch

    warps = torch.cuda.get_device_properties(0).multi_processor_count * 16
    return next((v for v in (1, 2, 4, 8, 16) if n <= v * warps), 32)


def _run(n, mode, opts):
    from loom_b200 import api

    table, want = _scene(n)
    with api.Function("sphere_pt_f32", n, mode, **opts) as f:
        got = f.launch_host([api.Broadcast(0, "u32"), api.Iota()], n, table=table)
        s = f.stats(raise_on_device_error=True)
    for g, w in zip(got, want):
        assert np.array_equal(g.view(np.uint32), np.asarray(w).view(np.uint32))
    assert s["threads"] == n
    return s["grid"]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 16 * 148, 16 * 148 + 1, 4 * 16 * 148 + 5, 16 * 16 * 148, 16 * 16 * 148 + 1])
@pytest.mark.parametrize("mode,opts", [("plain", {}), ("plain", dict(block_size=100)),
                                       ("regroup", dict(plain_below=1 << 40, block_size=512))])
def test_large_kernel(n, mode, opts):
    assert _run(n, mode, opts) == -(-n // _lanes(n))


@pytest.mark.parametrize("n", [33, 257])
def test_large_kernel_at_a_named_size(n):
    assert _run(n, "plain", dict(block_size=256)) == -(-n // 256)


@pytest.mark.parametrize("n", [1, 33, 4735, 4737, 50000, 151553])
@pytest.mark.parametrize("opts", [dict(), dict(schedule=2, period=0xFFFFFFFF, prefetch=False, max_regs=56, refill_lanes=10),
                                  dict(schedule=2, burst=4, period=9, population=300), dict(schedule=3, period=64),
                                  dict(cost_model=True, refill=False)])
def test_fewer_threads_than_lanes(n, opts):
    """The megakernel's warps take their share of a small launch."""
    _run(n, "regroup", opts)


@pytest.mark.parametrize("opts,cta", [({}, 256), (dict(block_size=64), 64)])
def test_small_kernel(opts, cta):
    from loom_b200 import api
    from oracle import oracle as O

    x = np.arange(1, 1001, dtype=np.uint64)
    (want,) = O.Interp("collatz_u64").run([x])
    with api.Function("collatz_u64", 1000, "plain", **opts) as f:
        assert np.array_equal(f(x), want)
        assert f.stats()["grid"] == -(-1000 // cta)
