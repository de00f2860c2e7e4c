"""Table records read through one address (the generator's rows): the rows
of hand-written blocks (CPU), and, on the GPU, launches whose table is flat,
declared too large to be, of unstated size, and not 16-byte aligned, which
all give the oracle's bits."""

import ctypes

import numpy as np
import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir

HEAD = """loomir 1
kernel t
index u32
straight 1
reg 0 a 4 u32
reg 1 b 4 u32
reg 2 x 4 f32
reg 3 y 4 f32
reg 4 z 4 f32
input 0 u32 a
output 2 f32 x
block 0 START 9
"""


def _rows(body):
    k = ir.parse(HEAD + body + "end\n")
    return E.Lowering(k).table_rows(k.blocks[0].instrs)


def test_row_of_fields_in_any_order():
    rows, member = _rows(
        "i add u32 r1:u32 r0:u32 ku32:0x3\n"
        "i tab f32 r2:f32 r1:u32\n"
        "i add u32 r1:u32 ku32:0x1 r0:u32\n"
        "i tab f32 r3:f32 r1:u32\n"
        "i mov - r1:u32 r0:u32\n"
        "i add u32 r1:u32 r1:u32 ku32:0x8\n"
        "i tab f32 r4:f32 r1:u32\n"
    )
    # lowest read: a + 1, reached from the first read's index a + 3
    assert rows == {1: ("R.r1 - 2u", [0, 2, 7])}
    assert member == {1: (1, 2), 3: (1, 0), 6: (1, 7)}


def test_row_ends_at_its_span_and_at_a_changed_index():
    rows, member = _rows(
        "i tab f32 r2:f32 r0:u32\n"
        f"i add u32 r1:u32 r0:u32 ku32:{E.ROW_SPAN:#x}\n"
        "i tab f32 r3:f32 r1:u32\n"
        f"i add u32 r1:u32 r0:u32 ku32:{E.ROW_SPAN + 1:#x}\n"
        "i tab f32 r4:f32 r1:u32\n"
        "i mul u32 r0:u32 r0:u32 ku32:0x2\n"  # another value from here on
        "i tab f32 r2:f32 r0:u32\n"
    )
    assert rows == {0: ("R.r0", [0, E.ROW_SPAN])}
    assert member == {0: (0, 0), 2: (0, E.ROW_SPAN)}


def test_single_reads_form_no_row():
    rows, member = _rows("i tab f32 r2:f32 r0:u32\ni mul u32 r0:u32 r0:u32 ku32:0x2\ni tab f32 r3:f32 r0:u32\n")
    assert rows == {} and member == {}


@pytest.mark.gpu
@pytest.mark.parametrize("opts", [dict(), dict(schedule=2, period=0xFFFFFFFF, prefetch=False, max_regs=56)])
@pytest.mark.parametrize("mode", ["plain", "regroup"])
def test_flat_and_other_tables_give_the_same_bits(mode, opts):
    import torch

    from loom_b200 import api
    from loom_b200 import scenes as S
    from oracle import oracle as O

    req = S.cornell_request(37, 21, 4, seed=3)
    table, _ = S.pack([req])
    n = req.threads
    want = O.Interp("sphere_pt_f32").run([np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32)], table=table)
    for shift in (0, 1):  # words from a 16-byte boundary
        d = torch.zeros(len(table) + shift, dtype=torch.int32, device="cuda")
        d[shift:] = torch.from_numpy(table.view(np.int32)).cuda()
        for words in (len(table), 0, 0xFFFFFFFF):  # flat; unstated; declared above the flat limit
            out = [torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3)]
            with api.Function("sphere_pt_f32", 0, mode, **opts) as f:
                L, keep = f._launch_struct([api.Broadcast(0, "u32"), api.Iota()], out, n, None, d[shift:])
                L.table_words = words
                api.check(api.lib().loom_b200_launch_device(f._h, ctypes.byref(L), None))
                f.stats(raise_on_device_error=True)
                del keep
            for g, w in zip(out, want):
                assert np.array_equal(g.cpu().numpy().view(np.uint32), np.asarray(w).view(np.uint32))
