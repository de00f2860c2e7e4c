"""Selections among constants that become rows of constant memory: grouping
and the tables' words, for hand-written blocks and every registry kernel
(CPU; the path tracers' own parity tests run them on the GPU)."""

import pathlib
import re

import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir

GEN = pathlib.Path(__file__).resolve().parents[1] / "loom_b200" / "csrc" / "gen"
HEAD = "loomir 1\nkernel t\nindex u32\nstraight 1\nreg 0 i 4 u32\nreg 1 a 4 f32\nreg 2 b 4 f32\nreg 3 c 4 u32\nreg 4 j 4 i32\ninput 0 u32 i\noutput 1 f32 a\nblock 0 START 9\n"


def _rows(body):
    k = ir.parse(HEAD + body + "end\n")
    L = E.Lowering(k)
    return L.constant_rows(k.blocks[0].instrs), L.constant_tables(k.blocks[0])


A = "i sct f32,u32 r1:f32 r0:u32 | kf32:0x1 kf32:0x2 kf32:0x3\n"
B = "i sct f32,u32 r2:f32 r0:u32 | kf32:0x4 kf32:0x5 kf32:0x6\n"
C = "i sct u32,u32 r3:u32 r0:u32 | ku32:0x7 ku32:0x8 ku32:0x9\n"


def test_a_row_of_three():
    rows, tables = _rows(A + B + C)
    assert [(n, ps) for _, n, ps in rows.values()] == [(3, [0, 1, 2])]
    assert tables == ["__constant__ uint4 kSct0_0[3] = {{0x1u, 0x4u, 0x7u, 0u}, {0x2u, 0x5u, 0x8u, 0u}, {0x3u, 0x6u, 0x9u, 0u}};"]


@pytest.mark.parametrize(
    "body",
    [
        A + B,  # too few
        A + "i add u32 r0:u32 r0:u32 ku32:0x1\n" + B + C,  # the index changes
        A + B + "i sct u32,u32 r3:u32 r0:u32 | ku32:0x7 ku32:0x8\n",  # other entries
        (A + B + C).replace("r0:u32", "r4:i32").replace(",u32", ",i32"),  # a signed index is not clamped
    ],
)
def test_what_forms_no_row(body):
    assert _rows(body) == ({}, [])


@pytest.mark.parametrize("name", ["pt_const_512", "pt2_const_40", "primary_const_256"])
def test_tables_of_the_registry(name):
    """Word j of entry i is the i-th constant of the row's j-th selection."""
    k = ir.load(name)
    L = E.Lowering(k)
    src = (GEN / f"{name}.cu").read_text()
    found = 0
    for b in k.blocks:
        for first, (idx, n, ps) in L.constant_rows(b.instrs).items():
            m = re.search(rf"__constant__ uint4 kSct{b.idx}_{first}\[(\d+)\] = \{{(.*)\}};", src)
            words = [int(x, 16) if x.startswith("0x") else int(x) for x in re.findall(r"(0x[0-9a-f]+|\d+)u", m.group(2))]
            width = (len(ps) + 3) // 4 * 4
            assert int(m.group(1)) * 4 == len(words) == n * width
            for j, p in enumerate(ps):
                assert [words[i * width + j] for i in range(n)] == [c.bits for c in b.instrs[p].consts]
            found += 1
    assert found >= 3
