"""Self-loops run in groups of copies: which loops count (CPU), and launches
whose iteration counts lie around the group sizes, under step guards that
end inside a group (GPU), against the oracle."""

import numpy as np
import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir


def _loop(body, stay="1 0", typ="u32"):
    head = f"loomir 1\nkernel t\nindex u32\nstraight 0\nreg 0 i 4 {typ}\nreg 1 n 4 {typ}\nreg 2 c 4 u32\nreg 3 x 4 f32\n"
    text = f"input 0 {typ} i\ninput 1 {typ} n\noutput 3 f32 x\nblock 0 loop 4\n{body}p r2:u32 {stay}\nend\n"
    return ir.parse(head + text.replace("1 0", "-1 0")).blocks[0]


STEP = "i add u32 r0:u32 r0:u32 ku32:0x1\n"


@pytest.mark.parametrize(
    "body,cmp",
    [
        (STEP + "i lt u32 r2:u32 r0:u32 r1:u32\n", "lt"),
        (STEP + "i ge u32 r2:u32 r1:u32 r0:u32\n", "le"),
        (STEP + "i ne u32 r2:u32 r0:u32 ku32:0x7\n", "ne"),
        ("i gt f32 r2:u32 r3:f32 kf32:0x0\n" + STEP + "i le u32 r2:u32 r0:u32 r1:u32\n", "le"),
        ("i lt u32 r2:u32 r0:u32 r1:u32\n" + STEP, None),  # compared before the step
        (STEP + "i add u32 r1:u32 r1:u32 r1:u32\ni lt u32 r2:u32 r0:u32 r1:u32\n", None),  # the bound moves
        (STEP + STEP + "i lt u32 r2:u32 r0:u32 r1:u32\n", None),  # two steps
        (STEP.replace("0x1", "0x2") + "i lt u32 r2:u32 r0:u32 r1:u32\n", None),
        (STEP + "i gt u32 r2:u32 r0:u32 r1:u32\n", None),  # goes on above the bound
        (STEP + "i lt u32 r2:u32 r0:u32 r1:u32\ni land u32 r2:u32 r2:u32 r1:u32\n", None),  # not the last word
    ],
)
def test_counted_loops(body, cmp):
    got = E.counted_loop(_loop(body))
    assert (got and got[2]) == cmp


def test_registry_loops():
    want = {"collatz_u64": (None, 8), "fib_u64": ("le", 8), "fib_u32": ("le", 8), "sphere_pt_f32": ("lt", 4)}
    for name, (cmp, copies) in want.items():
        b = next(b for b in ir.load(name).blocks if b.idx in b.successors())
        got = E.counted_loop(b)
        assert (got and got[2]) == cmp and E.unroll_factor(b) == copies


GUARDS = [dict(), dict(max_steps=1), dict(max_steps=7), dict(max_steps=8), dict(max_steps=9), dict(max_steps=23)]


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["fib_u64", "fib_u32", "collatz_u64", "fac_u64"])
def test_iteration_counts_around_the_groups(kernel):
    from loom_b200 import api
    from oracle import oracle as O

    dt = api.NP_TYPE[api.info(kernel).inputs[0][1]]
    x = np.arange(0 if kernel != "collatz_u64" else 1, 94, dtype=dt)
    if kernel == "fac_u64":
        x = x[:21]
    (want,) = O.Interp(kernel).run([x])
    for mode, opts in [("plain", {}), ("regroup", {})] + [
        ("regroup", dict(schedule=2, period=0xFFFFFFFF, prefetch=False, burst=2, spin_iters=s)) for s in (1, 3, 16, 64, 0)
    ] + [("regroup", dict(burst=b, period=4)) for b in (1, 3, 8, 9)]:
        with api.Function(kernel, len(x), mode, **opts) as f:
            got = f(x)
            f.stats(raise_on_device_error=True)
        assert np.array_equal(got, want), (mode, opts)


@pytest.mark.gpu
@pytest.mark.parametrize("opts", GUARDS)
def test_step_guard_stops_inside_a_group(opts):
    """fib(n) enters its loop n - 1 times: threads within the guard halt
    with their result, one beyond it raises the step-limit status."""
    from loom_b200 import api

    most = opts.get("max_steps", 93)
    fib = [0, 1]
    while len(fib) < 94:
        fib.append(fib[-1] + fib[-2])
    within = np.arange(0, min(most + 2, 94), dtype=np.uint64)
    with api.Function("fib_u64", 94, "plain", **opts) as f:
        assert f(within).tolist() == [fib[int(v)] for v in within]
        f.stats(raise_on_device_error=True)
        if most + 2 < 94:
            x = np.append(within, np.uint64(most + 2))
            with pytest.raises(api.LoomError):
                f(x)
            assert f.stats()["status"] & api.STATUS_STEP_LIMIT
