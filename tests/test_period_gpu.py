"""What a tile may run in one round of the megakernel: `period` steps, the
iterations of a loop on one block among them, so that a launch stopped after
`max_steps` rounds has run no thread further than both allow (against counts
of the oracle)."""

import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPHERES = 208
ISECT = 38  # instructions of an iteration of the intersection loop


@functools.lru_cache(maxsize=None)
def _scene(n):
    """The Cornell box with one small sphere many times over, the oracle's
    outputs, and the intersection iterations of the longest of n paths: the
    copies change no path, so twice as many cost ISECT instructions each and
    pass."""
    from loom_b200 import scenes as S
    from oracle import oracle as O

    ins = [np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32)]
    counts = []
    for spheres in (SPHERES // 2, SPHERES):
        r = S.cornell_request(16, 16, 2, seed=9)
        r.spheres = (r.spheres + [r.spheres[-2]] * spheres)[:spheres]
        table, _ = S.pack([r])
        want, count = O.Interp("sphere_pt_f32").run(ins, table=table, count_instr=True)
        counts.append(count.astype(np.int64))
    passes, left = np.divmod(counts[1] - counts[0], ISECT * (SPHERES // 2))
    assert not left.any()
    return table, want, int(passes.max()) * SPHERES


@pytest.mark.parametrize("n", [32, 300])
@pytest.mark.parametrize("opts", [dict(period=32), dict(period=64, burst=8), dict(period=48, burst=16, schedule=1),
                                  dict(period=256), dict(period=32, spread_lanes=8, utr_lanes=1)])
def test_rounds_cover_the_iterations_run(n, opts):
    from loom_b200 import api

    table, want, iterations = _scene(n)
    ins = [api.Broadcast(0, "u32"), api.Iota()]
    enough = iterations // opts["period"]
    with api.Function("sphere_pt_f32", n, "regroup", **opts) as f:
        got = f.launch_host(ins, n, table=table)
        s = f.stats(raise_on_device_error=True)
    assert all(g.tobytes() == w.tobytes() for g, w in zip(got, want))
    assert s["rounds"] >= enough
    # stopped well before: the step guard speaks up
    with api.Function("sphere_pt_f32", n, "regroup", max_steps=max(1, enough // 2), **opts) as f:
        with pytest.raises(api.LoomError):
            f.launch_host(ins, n, table=table)
        assert f.stats()["status"] & api.STATUS_STEP_LIMIT
