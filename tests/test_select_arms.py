"""64-bit selects with a predicated arm (the generator's select_arms): random
blocks give the same live values when one arm's PTX, read back by a small
interpreter, runs over the other arm's result (CPU)."""

import random
import re

import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir
from loom_b200.codegen.ir import Compute, Operand

REGS = 7
MASK = (1 << 64) - 1
STORAGE = {i: "u64" for i in range(REGS)}
FN = {"add": lambda a, b: a + b, "sub": lambda a, b: a - b, "mul": lambda a, b: a * b, "band": lambda a, b: a & b,
      "bor": lambda a, b: a | b, "bxor": lambda a, b: a ^ b, "shr": lambda a, b: a >> (b & 63), "lt": lambda a, b: int(a < b)}
PTX = {v: FN[k] for k, v in E.PTX_OP.items()}


def _operand(rng):
    if rng.random() < 0.25:
        return Operand("u64", bits=rng.choice([0, 1, 3, MASK, 1 << 33]))
    return Operand("u64", reg=rng.randrange(REGS))


def _block(rng):
    out = []
    for _ in range(rng.randint(3, 10)):
        dst = Operand("u64", reg=rng.randrange(REGS))
        op = rng.choice(["add", "sub", "mul", "mul", "add", "band", "bor", "bxor", "shr", "lt", "cmov", "cmov"])
        if op == "cmov":
            out.append(Compute(op, (), dst, [_operand(rng) for _ in range(3)], []))
        else:
            out.append(Compute(op, ("u64",), dst, [_operand(rng), _operand(rng)], []))
        if op == "mul" and rng.random() < 0.7:  # the products that sums read
            out.append(Compute("add", ("u64",), dst, [dst, _operand(rng)], []))
            out.append(Compute("cmov", (), Operand("u64", reg=rng.randrange(REGS)), [_operand(rng), dst, _operand(rng)], []))
    return out


def _value(a, R):
    return a.bits if a.is_literal else R[a.reg]


def _run(ins, R):
    v = [_value(a, R) for a in ins.args]
    R[ins.dst.reg] = (v[1] if v[0] else v[2]) if ins.op == "cmov" else FN[ins.op](*v) & MASK


def _predicated(text, v, regs, R):
    """What the PTX leaves in %0 when its predicate holds."""
    t = {"%0": v, **{f"%{2 + i}": R[r] for i, r in enumerate(regs)}}
    for line in re.findall(r"@p ([^;]*);", text):
        op, rest = line.split(" ", 1)
        dst, *args = [x.strip() for x in rest.split(",")]
        a = [t[x] if x in t else int(x, 16) for x in args]
        t[dst] = (a[0] * a[1] + a[2] if op == "mad.lo.u64" else PTX[op](*a)) & MASK
    return t["%0"]


def test_random_selects_keep_every_live_value():
    rng = random.Random(7)
    seen = inverted_seen = fused = 0
    for _ in range(20000):
        block = _block(rng)
        live = set(rng.sample(range(REGS), rng.randint(0, 3)))
        arms = E.select_arms(block, live, STORAGE)
        if not arms:
            continue
        moved = {p for a, b, _ in arms.values() for p in a + b}
        for _ in range(5):
            R0 = [rng.choice([0, 1, 2, MASK, rng.getrandbits(64)]) for _ in range(REGS)]
            want, got = list(R0), list(R0)
            for ins in block:
                _run(ins, want)
            for p, ins in enumerate(block):
                if p in moved:
                    continue
                if p not in arms:
                    _run(ins, got)
                    continue
                line, asm, inverted = arms[p]
                for x in line:
                    _run(block[x], got)
                c = bool(_value(ins.args[0], got))
                v = _value(ins.args[1 if inverted else 2], got)
                text, regs = E.predicated_ptx([block[x] for x in asm])
                seen += 1
                inverted_seen += inverted
                fused += "mad" in text
                if c != inverted:
                    v = _predicated(text, v, regs, got)
                got[ins.dst.reg] = v
            # values computed for a select alone are dead after it
            for r in live:
                assert got[r] == want[r], (block, live, arms, R0, r)
    assert seen > 2000 and inverted_seen > 100 and fused > 100


@pytest.mark.parametrize("name,count", [("collatz_u64", 1), ("fib_u64", 0), ("sphere_pt_f32", 0)])
def test_registry_selects(name, count):
    k = ir.load(name)
    lo = k.liveness()[1]
    st = {r.idx: r.storage for r in k.regs}
    assert sum(len(E.select_arms(b.instrs, lo[b.idx], st)) for b in k.blocks) == count
