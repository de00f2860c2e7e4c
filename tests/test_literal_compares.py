"""64-bit compares with small literals: the operand is converted to the
compare's own type first, as every compare does, and only integer literals
take the form (CPU)."""

import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir

REGS = {"u64": 8, "i64": 8, "u32": 4, "i32": 4, "i8": 1, "f32": 4, "f64": 8}
HEAD = "loomir 1\nkernel t\nindex u32\nstraight 1\n" + "".join(f"reg {i} x{i} {n} {t}\n" for i, (t, n) in enumerate(REGS.items()))


def _expr(line):
    k = ir.parse(HEAD + "output 0 u64 x0\nblock 0 START 1\n" + line + "\nend\n")
    return E.Lowering(k, device=True).expr(k.blocks[0].instrs[0])


@pytest.mark.parametrize("t", ["u64", "i64"])
@pytest.mark.parametrize("a", list(REGS))
def test_operand_conversion(t, a):
    """A float's (or a narrow signed integer's) way to 64 bits is through the
    compare's type: -1.0f is -1 as i64, and no u64."""
    r = list(REGS).index(a)
    e = _expr(f"i ne {t} r0:u64 r{r}:{a} k{t}:0x5")
    wide = {"u64": "unsigned long long", "i64": "long long"}[t]
    assert e == f"op_differs(static_cast<unsigned long long>(static_cast<{wide}>(R.r{r})), 0x5u)"


@pytest.mark.parametrize("lit", ["kf32:0x3f800000", "kf64:0x3ff0000000000000", "ki64:0xffffffffffffffff", "ku64:0x100000000"])
def test_other_literals_take_the_plain_compare(lit):
    assert "op_differs" not in _expr(f"i eq i64 r0:u64 r1:i64 {lit}")
