"""Programs without loops at several Loom threads per CUDA thread: sizes
around the rule's line and the CTAs' edges, in place, against the oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

def _sample(n):
    """Threads to compare: the ends, CTA edges at both ends, and random ones."""
    rng = np.random.default_rng(n)
    at = [np.arange(min(n, 2100)), np.arange(max(0, n - 2100), n), rng.integers(0, n, 4000)]
    return np.unique(np.concatenate(at))


FILL = 148 * 2048 * 4  # threads from which several run per CUDA thread (148 SMs)


@pytest.mark.parametrize("n", [FILL - 1, FILL, FILL + 257, FILL + 1023])
@pytest.mark.parametrize("in_place", [False, True])
def test_threefry(n, in_place):
    import torch

    from loom_b200 import api
    from oracle import oracle as O

    rng = np.random.default_rng(n)
    x = [rng.integers(0, 1 << 32, n, dtype=np.uint32) for _ in range(2)]
    at = _sample(n)
    want = O.Interp("threefry_u32").run([a[at] for a in x])
    d = [torch.from_numpy(a.view(np.int32)).cuda() for a in x]
    out = d if in_place else [torch.full_like(a, -1) for a in d]
    with api.Function("threefry_u32", 0, "plain") as f:
        f.run_device(d, out, n)
        s = f.stats(raise_on_device_error=True)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per = 4 if n >= sms * 2048 * 4 else 1
    assert s["grid"] == -(-n // (256 * per)) and s["threads"] == n
    for g, w in zip(out, want):
        assert np.array_equal(g.cpu().numpy().view(np.uint32)[at], np.asarray(w))


@pytest.mark.parametrize("kernel", ["cross_f32", "arithmetic_f64", "increment_i16", "increment_u8"])
def test_types_and_input_forms(kernel):
    """Every width, with one broadcast column, past one full group of CTAs."""
    import torch

    from loom_b200 import api
    from oracle import oracle as O

    n = FILL + 777
    info = api.info(kernel)
    rng = np.random.default_rng(4)
    dt = [api.NP_TYPE[t] for _, t in info.inputs]
    x = [rng.uniform(0.5, 2, n).astype(t) if np.dtype(t).kind == "f" else rng.integers(0, 100, n).astype(t) for t in dt]
    forms = list(x)
    if len(x) > 1:
        forms[-1] = api.Broadcast(x[-1][0], info.inputs[-1][1])
        x[-1] = np.full(n, x[-1][0], dtype=dt[-1])
    at = _sample(n)
    want = O.Interp(kernel).run([a[at] for a in x])
    with api.Function(kernel, n, "plain", host_chunks=1) as f:
        got = f.launch_host(forms, n)
        f.stats(raise_on_device_error=True)
    for g, w in zip(got if isinstance(got, tuple) else [got], want):
        assert np.array_equal(np.ascontiguousarray(np.asarray(g)[at]).view(np.uint8), np.ascontiguousarray(w).view(np.uint8))
