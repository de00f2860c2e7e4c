"""Tables of unstated size in device launches: the allocation bounds them, or,
where an allocator maps memory piece by piece into a large reservation, the
reservation, never one piece.  Seen from the grid: at 40 registers a flat
table's launch keeps more CTAs on an SM than one on any other table, which
runs at the default register cap."""

import os
import pathlib
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = pathlib.Path(__file__).resolve().parents[1]

BODY = """
import ctypes
import torch
import numpy as np
from loom_b200 import api, scenes as S

table, _ = S.pack([S.cornell_request(16, 16, 2, seed=9)])
n = 512
d = torch.from_numpy(table.view(np.int32)).cuda()
out = [torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3)]
grid = []
for words in (len(table), 0xFFFFFFFF, 0):
    with api.Function("sphere_pt_f32", 0, "regroup", schedule=1, cost_model=True, block_size=512, max_regs=40, population=4096) as f:
        L, keep = f._launch_struct([api.Broadcast(0, "u32"), api.Iota()], out, n, None, d)
        L.table_words = words
        api.check(api.lib().loom_b200_launch_device(f._h, ctypes.byref(L), None))
        grid.append(f.stats(raise_on_device_error=True)["grid"])
print(*grid)
"""


@pytest.mark.parametrize("pieces", [False, True])
def test_unstated_table_sizes(pieces):
    env = dict(os.environ, PYTORCH_CUDA_ALLOC_CONF=f"expandable_segments:{pieces}")
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(BODY)], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    flat, other, unstated = map(int, r.stdout.split()[-3:])
    assert flat > other
    assert unstated == (other if pieces else flat)
