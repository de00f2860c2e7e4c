"""Programs whose steps of schedule 2 need no order: one loop at most, and no
long block for which lanes may have to wait (opts.defer_lanes) (CPU)."""

import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir


def _kernel(*blocks):
    """Blocks as (instructions, terminator)."""
    text = "loomir 1\nkernel t\nindex u32\nstraight 0\nreg 0 n 4 u32\ninput 0 u32 n\noutput 0 u32 n\n"
    for i, (n, term) in enumerate(blocks):
        text += f"block {i} b{i} {n + 1}\n" + "i add u32 r0:u32 r0:u32 ku32:0x1\n" * n + term + "\n"
    return ir.parse(text + "end\n")


LONG = E.LONG_BLOCK_INSTR
LOOP = "p r0:u32 -1 1"


@pytest.mark.parametrize(
    "blocks,free",
    [
        ([(2, "j -1")], True),  # no loop
        ([(LONG, "j -1")], True),  # every lane at block 0
        ([(2, "j 1"), (2, LOOP)], True),  # one short loop
        ([(LONG, "p r0:u32 -1 0")], True),  # one block for all lanes
        ([(2, "j 1"), (LONG, LOOP)], False),  # lanes may wait at the loop
        ([(LONG, "j 1"), (2, LOOP)], False),  # ... or before it
        ([(2, "j 1"), (2, "j 2"), (LONG, "p r0:u32 -1 1")], True),  # the long block is no place to stand
        ([(2, "j 1"), (2, "p r0:u32 2 1"), (2, "p r0:u32 -1 2")], False),  # two loops
    ],
)
def test_programs_without_order(blocks, free):
    k = _kernel(*blocks)
    assert f"kAnyOrder = {str(free).lower()};" in E.generate(k)


@pytest.mark.parametrize("name,free", [("collatz_u64", True), ("fib_u32", True), ("threefry_u32", True), ("sphere_pt_f32", False), ("pt_const_40", False)])
def test_the_registry(name, free):
    assert E.any_order(ir.load(name)) == free
