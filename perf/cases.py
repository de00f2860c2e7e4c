"""Timed cases: what users of this framework run, through its public entry
points, from the smallest launch to the headline render.

Every case is one call (or a short fixed sequence of calls) on handles that
a user's program keeps: integer loop kernels and random numbers on device
columns, the drop-in host call, the sphere path tracer in its tuned, default
and lane-efficiency forms, images as per-pixel means, batched render
requests, Loom's own path tracer, and the continuous-batching servers.
Options come from the shipped tuning table or are the defaults, as in the
documentation's examples.
"""

import math

import numpy as np
import torch

from loom_b200 import api
from loom_b200 import autotune
from loom_b200 import scenes as S
from loom_b200 import serving

FORMS = {
    # the regrouping engine at the options tuned for one large render
    "tuned": ("regroup", "pt"),
    # the same engine held to a high SIMT lane efficiency (parks threads)
    "lane": ("regroup", "pt_lane"),
    # Loom's majority rule with the cost model (parks threads)
    "majority": ("regroup", "pt_majority"),
    # a handle made without any option
    "default": ("regroup", None),
    # the drop-in engine, one CUDA thread per Loom thread
    "plain": ("plain", None),
}


def listed():
    return [
        # a small host-driven step: one launch of a few warps, where the call counts
        {"name": "fib_1k", "kind": "loop", "kernel": "fib_u64", "n": 1000, "form": "plain"},
        # Loom's README example at the size of its benchmarks
        {"name": "fib_1m", "kind": "loop", "kernel": "fib_u64", "n": 1 << 20, "form": "tuned"},
        # the divergent integer loop, a full GPU of it
        {"name": "collatz_16m", "kind": "loop", "kernel": "collatz_u64", "n": 1 << 24, "form": "tuned"},
        # the drop-in call on host arrays with default options (README usage), an odd size
        {"name": "collatz_host_1m", "kind": "host_loop", "kernel": "collatz_u64", "n": 1000003},
        # counter-based random-number columns: a straight-line kernel, streaming
        {"name": "threefry_20m", "kind": "threefry", "n": 20000003},
        # the headline render with its image
        {"name": "pt_image", "kind": "render", "w": 1024, "h": 768, "spp": 64, "form": "tuned", "image": True},
        # a render request end to end: host table in, image on the host, odd sizes
        {"name": "pt_image_host", "kind": "render_host", "w": 500, "h": 333, "spp": 16},
        # a preview render as the command-line tool makes it, default options
        {"name": "pt_default", "kind": "render", "w": 320, "h": 240, "spp": 16, "form": "default", "image": False},
        # a mid-size render in the lane-efficiency form
        {"name": "pt_lane", "kind": "render", "w": 512, "h": 384, "spp": 16, "form": "lane", "image": False},
        # uneven render requests in one launch (8-64 spheres each)
        {"name": "batch_48", "kind": "batch", "requests": 48, "mix": 3},
        # Loom's own path tracer, a 384 x 384 window of its 512 x 512 image
        {"name": "loom_pt", "kind": "loom", "w": 384, "h": 384, "form": "plain"},
        # a burst of mixed requests through the continuous-batching servers
        {"name": "serve_32", "kind": "serve", "requests": 32, "mix": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "loop", "host_loop", "threefry", "render", "render", "render", "render_host",
                       "batch", "loom", "serve"])
    if kind == "loop":
        kernel = rng.choice(["fib_u64", "collatz_u64"])
        n = _log(rng, 1000, (1 << 20) if kernel == "fib_u64" else (1 << 24))
        return {"kind": kind, "kernel": kernel, "n": n, "form": rng.choice(["tuned", "default", "plain"])}
    if kind == "host_loop":
        return {"kind": kind, "kernel": rng.choice(["fib_u64", "collatz_u64"]), "n": _log(rng, 1000, 1000003)}
    if kind == "threefry":
        return {"kind": kind, "n": _log(rng, 1000, 20000003)}
    if kind in ("render", "render_host"):
        form = rng.choice(sorted(FORMS)) if kind == "render" else "tuned"
        # pixels and samples over their ranges, up to the headline's threads
        # for the tuned form and a sixteenth of them for the slower ones
        most = (1024 * 768 * 64) if form == "tuned" and kind == "render" else 1024 * 768 * 4
        w, h, spp = _log(rng, 31, 1024), _log(rng, 23, 768), 1 << rng.randint(0, 6)
        while w * h * spp > most:
            spp //= 2
        if kind == "render_host":
            return {"kind": kind, "w": w, "h": h, "spp": spp}
        return {"kind": kind, "w": w, "h": h, "spp": spp, "form": form, "image": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "requests": rng.randint(2, 48), "mix": rng.randint(10, 999999)}
    if kind == "loom":
        return {"kind": kind, "w": _log(rng, 17, 384), "h": _log(rng, 17, 384), "form": rng.choice(["tuned", "plain"])}
    return {"kind": kind, "requests": rng.randint(4, 32), "mix": rng.randint(10, 999999)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _loop_range(kernel):
    """fib: n in [0, 93], whose results fit in u64; collatz: n in [1, 2^32)."""
    return (0, 94) if kernel == "fib_u64" else (1, 1 << 32)


def _loop_out(kernel):
    return torch.int64 if kernel == "fib_u64" else torch.int32


def _opts(kernel, form, graph=False):
    """(mode, options) of a form: the shipped tuning, or none."""
    if form == "plain":
        return "plain", {}
    if form == "default":
        return "regroup", {}
    key = FORMS[form][1] if kernel == "sphere_pt_f32" else "default"
    return "regroup", dict(autotune.tuned(kernel, key), graph=graph)


def _mix(case):
    """Sizes of a batch's or a burst's render requests: resolution from
    {64, 128, 256, 512}^2, spp from {1, 4, 16, 64}.  They follow from the
    case alone; the scenes follow from the seed."""
    rng = np.random.default_rng(case["mix"])
    return [(int(rng.choice([64, 128, 256, 512])), int(rng.choice([1, 4, 16, 64])), rng.uniform(),
             int(rng.integers(16, 19))) for _ in range(case["requests"])]


def _random_scene(rng, res, spp, seed):
    r = S.random_request(rng, seed=seed)
    r.width, r.height, r.spp = res, res, spp
    return r


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("loop", "host_loop"):
        lo, hi = _loop_range(case["kernel"])
        n = case["n"]
        x = torch.randint(lo, hi, (n,), dtype=torch.int64, device="cuda", generator=_gen(seed))
        if kind == "host_loop":
            return {"kind": kind, "x": x.cpu().numpy().view(np.uint64), "f": api.Function(case["kernel"], n, "regroup")}
        mode, o = _opts(case["kernel"], case["form"])
        return {"kind": kind, "n": n, "x": x, "f": api.Function(case["kernel"], 0, mode, **o),
                "y": torch.empty(n, dtype=_loop_out(case["kernel"]), device="cuda")}
    if kind == "threefry":
        n, g = case["n"], _gen(seed)
        return {"kind": kind, "n": n, "f": api.Function("threefry_u32", 0, "plain"),
                "in": [torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=g)
                       for _ in range(2)],
                "out": [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]}
    if kind == "render":
        req = S.cornell_request(case["w"], case["h"], case["spp"], seed=seed)
        table, _ = S.pack([req])
        n, pixels = req.threads, case["w"] * case["h"]
        mode, o = _opts("sphere_pt_f32", case["form"], graph=case["form"] == "tuned")
        return {"kind": kind, "n": n, "pixels": pixels, "spp": case["spp"],
                "f": api.Function("sphere_pt_f32", 0, mode, **o),
                "ins": [api.Broadcast(0, "u32"), api.Iota()],
                "table": torch.from_numpy(table.view(np.int32)).cuda(),
                "out": [torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3)],
                "img": [torch.empty(pixels, dtype=torch.float32, device="cuda") for _ in range(3)] if case["image"] else None}
    if kind == "render_host":
        req = S.cornell_request(case["w"], case["h"], case["spp"], seed=seed)
        table, _ = S.pack([req])
        mode, o = _opts("sphere_pt_f32", "tuned")
        return {"kind": kind, "n": req.threads, "spp": case["spp"], "table": table,
                "f": api.Function("sphere_pt_f32", req.threads, mode, **o),
                "ins": [api.Broadcast(0, "u32"), api.Iota()],
                "img": [torch.empty(case["w"] * case["h"], dtype=torch.float32).pin_memory() for _ in range(3)]}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        reqs = [_random_scene(rng, res, spp, i + 1) for i, (res, spp, _, _) in enumerate(_mix(case))]
        table, starts = S.pack(reqs)
        n = int(starts[-1])
        o = dict(autotune.tuned("sphere_pt_f32", "batch"), graph=True)
        return {"kind": kind, "n": n, "f": api.Function("sphere_pt_f32", 0, "regroup", **o),
                "ins": [api.Instance(), api.LocalIota()],
                "table": torch.from_numpy(table.view(np.int32)).cuda(),
                "starts": torch.from_numpy(starts.view(np.int64)).cuda(),
                "out": [torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3)]}
    if kind == "loom":
        w, h = case["w"], case["h"]
        rng = np.random.default_rng(seed)
        # a window of the image; where it fills the image, its place says nothing
        x0, y0 = (int(rng.integers(0, 512 - d + 1)) for d in (w, h))
        x, y = np.meshgrid(np.arange(w, dtype=np.int32) + x0, np.arange(h, dtype=np.int32) + y0)
        mode, o = _opts("pt_const_512", case["form"])
        n = w * h
        return {"kind": kind, "n": n, "f": api.Function("pt_const_512", 0, mode, **o),
                "in": [torch.from_numpy(((x << 16) | y).reshape(-1)).cuda()],
                "out": [torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3)]
                + [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2)]}
    return _prepare_serve(case, seed)


def _serve_sizes(case):
    """(kind, threads, resolution, spp) of each request of a burst: 60 %
    renders (at most 256^2 pixels at 16 samples, so that the burst stays a
    short one), 20 % collatz and 20 % fib batches of 2^16 to 2^18 inputs."""
    out = []
    for res, spp, u, lg in _mix(case):
        if u < 0.6:
            res, spp = min(res, 256), min(spp, 16)
            out.append(("pt", res * res * spp, res, spp))
        else:
            out.append(("collatz" if u < 0.8 else "fib", 1 << lg, 0, 0))
    return out


def _prepare_serve(case, seed):
    rng, g = np.random.default_rng(seed), _gen(seed)
    sizes = _serve_sizes(case)
    total = {k: max(1, sum(n for kk, n, _, _ in sizes if kk == k)) for k in ("pt", "collatz", "fib")}
    budget = api.Budget(8 << 30)
    pool = serving.Pool({
        "pt": api.Server("sphere_pt_f32", ring_threads=1 << 22, max_requests=64, slice_rounds=4,
                         forms=["instance", "local_iota"], header_words=S.HEADER_WORDS, reloc_word=4,
                         table_words=1 << 16, budget=budget, **autotune.tuned("sphere_pt_f32", "serve")),
        "collatz": api.Server("collatz_u64", ring_threads=1 << 22, max_requests=64, slice_rounds=2, budget=budget,
                              **{**autotune.tuned("collatz_u64", "serve"), "population": 1 << 20}),
        "fib": api.Server("fib_u64", ring_threads=1 << 22, max_requests=64, slice_rounds=2, budget=budget,
                          **{**autotune.tuned("fib_u64"), "population": 1 << 20, "block_size": 256, "ctas_per_sm": 0}),
    })
    outs = {"pt": [torch.empty(total["pt"], dtype=torch.float32).pin_memory() for _ in range(3)],
            "collatz": [torch.empty(total["collatz"], dtype=torch.int32).pin_memory()],
            "fib": [torch.empty(total["fib"], dtype=torch.int64).pin_memory()]}
    for cols in outs.values():
        for c in cols:
            c.zero_()
    pools = {k: torch.randint(*_loop_range(kern), (total[k],), dtype=torch.int64, device="cuda", generator=g).cpu().pin_memory()
             for k, kern in (("collatz", "collatz_u64"), ("fib", "fib_u64"))}
    at = {k: 0 for k in outs}
    reqs = []
    for i, (k, n, res, spp) in enumerate(sizes):
        o = [c[at[k]:at[k] + n] for c in outs[k]]
        if k == "pt":
            header, body = S.request_words(_random_scene(rng, res, spp, i + 1))
            reqs.append((k, n, dict(outputs=o, header=header, body=body)))
        else:
            reqs.append((k, n, dict(outputs=o, inputs=[pools[k][at[k]:at[k] + n]])))
        at[k] += n
    return {"kind": "serve", "pool": pool, "reqs": reqs, "outs": outs}


# ------------------------------------------------------------------ passes
def run(s):
    kind = s["kind"]
    if kind == "loop":
        s["f"].run_device([s["x"]], [s["y"]], s["n"])
        return s["y"]
    if kind == "host_loop":
        return s["f"](s["x"])
    if kind in ("threefry", "loom"):
        s["f"].run_device(s["in"], s["out"], s["n"])
        return s["out"]
    if kind == "render":
        s["f"].launch_device(s["ins"], s["out"], s["n"], table=s["table"])
        if s["img"] is None:
            return s["out"]
        for o, img in zip(s["out"], s["img"]):
            api.group_mean(o, img, s["pixels"], s["spp"])
        return s["out"] + s["img"]
    if kind == "render_host":
        return s["f"].launch_host_mean(s["ins"], s["n"], group=s["spp"], table=s["table"], outputs=s["img"])
    if kind == "batch":
        s["f"].launch_device(s["ins"], s["out"], s["n"], instance_starts=s["starts"], table=s["table"])
        return s["out"]
    for k, n, r in s["reqs"]:
        s["pool"].submit(k, n, **r)
    while s["pool"].busy():
        for key in s["pool"].step():
            s["pool"].result(*key)
    return s["outs"]


# ------------------------------------------------------------------ work
# Operations of a Loom thread: the program's own instructions, integer ones
# included, on average over the inputs (counted launches; a batched request's
# random scene takes about half of the Cornell box's).
OPS = {"fib_u64": 280, "collatz_u64": 1750, "threefry_u32": 200, "sphere_pt_f32": 6364, "pt_const_512": 2388000}
BATCH_OPS = 3260


def work(case):
    kind = case["kind"]
    if kind in ("loop", "host_loop"):
        return {"bytes": case["n"] * (16 if case["kernel"] == "fib_u64" else 12), "flops": case["n"] * OPS[case["kernel"]]}
    if kind == "threefry":
        return {"bytes": case["n"] * 16, "flops": case["n"] * OPS["threefry_u32"]}
    if kind in ("render", "render_host"):
        pixels = case["w"] * case["h"]
        n = pixels * case["spp"]
        # the samples leave the device only as their means in the host call
        out = 12 * pixels if kind == "render_host" else 12 * n + (12 * pixels if case["image"] else 0)
        return {"bytes": 352 + out, "flops": n * OPS["sphere_pt_f32"]}
    if kind == "batch":
        n = sum(res * res * spp for res, spp, _, _ in _mix(case))
        return {"bytes": 12 * n, "flops": n * BATCH_OPS}
    if kind == "loom":
        n = case["w"] * case["h"]
        return {"bytes": 24 * n, "flops": n * OPS["pt_const_512"]}
    b = f = 0
    for k, n, _, _ in _serve_sizes(case):
        b += n * {"pt": 12, "collatz": 12, "fib": 16}[k]
        f += n * {"pt": BATCH_OPS, "collatz": OPS["collatz_u64"], "fib": OPS["fib_u64"]}[k]
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ values
def _fib(x):
    t = [0, 1]
    while len(t) < 94:
        t.append(t[-1] + t[-2])
    t = np.array(t, dtype=np.uint64).view(np.int64)
    return torch.from_numpy(t).to(x.device)[x]


def _collatz(x):
    """Steps until n == 1, the threads still running kept dense."""
    steps = torch.zeros_like(x)
    at = torch.arange(len(x), device=x.device)
    v, k = x.clone(), 0
    while len(v):
        go = v > 1
        steps[at[~go]] = k
        at, v = at[go], v[go]
        v = torch.where((v & 1) == 1, 3 * v + 1, v >> 1)
        k += 1
    return steps.to(torch.int32)


def exact(case, seed):
    """Loop kernels only.  A path's radiance follows from its branches, which
    the kernels take in 32 bits: the same path in 64 bits is another one."""
    if case["kind"] not in ("loop", "host_loop"):
        return None
    lo, hi = _loop_range(case["kernel"])
    x = torch.randint(lo, hi, (case["n"],), dtype=torch.int64, device="cuda", generator=_gen(seed))
    y = (_fib if case["kernel"] == "fib_u64" else _collatz)(x)
    if case["kind"] == "host_loop":
        y = y.cpu().numpy()
        return y.view(np.uint64) if case["kernel"] == "fib_u64" else y.view(np.uint32)
    return y
