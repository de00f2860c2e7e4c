"""Work moved behind the condition it belongs to (the generator's guarded
regions): random branch-free blocks give the same live values in the
generated order as in program order, whatever the condition holds (CPU)."""

import random

import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir
from loom_b200.codegen.ir import Compute, Operand, ParmJump

REGS = 8
MASK = 0xFFFFFFFF


def _operand(rng):
    if rng.random() < 0.2:
        return Operand("u32", bits=rng.choice([0, 1, 2, 7]))
    return Operand("u32", reg=rng.randrange(REGS))


def _block(rng):
    out = []
    for _ in range(rng.randint(6, 24)):
        dst = Operand("u32", reg=rng.randrange(REGS))
        op = rng.choice(["lt", "ge", "pacc", "pacc", "land", "cmov", "cmov", "cmov", "add", "mul", "div", "mov"])
        a, b, c = _operand(rng), _operand(rng), _operand(rng)
        keep = rng.random() < 0.7  # the forms the analysis looks for
        if op == "pacc":
            out.append(Compute(op, ("u32", "u32", rng.choice(["land", "lor"]), "lt"), dst, [dst if keep else a, b, c], []))
        elif op == "cmov":
            out.append(Compute(op, (), dst, [a, b, dst if keep else c], []))
        elif op == "mov":
            out.append(Compute(op, (), dst, [a], []))
        else:
            out.append(Compute(op, ("u32",), dst, [dst if op == "land" and keep else a, b], []))
    return out + [ParmJump(Operand("u32", reg=rng.randrange(REGS)), [1, -1])]


def _run(ins, R):
    v = [R[a.reg] if not a.is_literal else a.bits for a in ins.args]
    op = ins.op
    if op == "pacc":
        c = v[1] < v[2]
        r = (bool(v[0]) and c) if ins.optype[2] == "land" else (bool(v[0]) or c)
    else:
        r = {
            "lt": lambda: v[0] < v[1],
            "ge": lambda: v[0] >= v[1],
            "land": lambda: bool(v[0]) and bool(v[1]),
            "cmov": lambda: v[1] if v[0] else v[2],
            "add": lambda: v[0] + v[1],
            "mul": lambda: v[0] * v[1],
            "div": lambda: v[0] // max(1, v[1]),
            "mov": lambda: v[0],
        }[op]()
    R[ins.dst.reg] = int(r) & MASK


def test_regions_of_random_blocks_keep_every_live_value():
    rng = random.Random(11)
    taken = skipped = 0
    for _ in range(6000):
        block = _block(rng)
        live = set(rng.sample(range(REGS), rng.randint(0, 4)))
        sink = E.guarded_region(block, live, set())
        if sink is None:
            continue
        cond, inside = sink
        assert all(cond < p < len(block) - 1 for p in inside)
        for _ in range(6):
            R0 = [rng.choice([0, 0, 1, 2, 5, MASK]) for _ in range(REGS)]
            want, got = list(R0), list(R0)
            for ins in block[:-1]:
                _run(ins, want)
            for ins in block[: cond + 1]:
                _run(ins, got)
            if got[block[cond].dst.reg]:
                taken += 1
                for p in sorted(inside):
                    _run(block[p], got)
            else:
                skipped += 1
            for p in range(cond + 1, len(block) - 1):
                if p not in inside:
                    _run(block[p], got)
            for r in live | set(block[-1].reads()):
                assert got[r] == want[r], (block, live, sink, R0, r)
    assert taken > 300 and skipped > 300


def test_a_small_region_stays_in_line():
    """Under SINK_MIN_COST the branch costs more than the work."""
    r = [Operand("u32", reg=i) for i in range(3)]
    block = [Compute("lt", ("u32",), r[0], [r[1], r[2]], []), Compute("add", ("u32",), r[1], [r[1], r[2]], []),
             Compute("cmov", (), r[2], [r[0], r[1], r[2]], [])]
    assert E.guarded_region(block, {2}, set()) is None


@pytest.mark.parametrize("name,label,op", [("sphere_pt_f32", "isect", "sqrt"), ("pt_const_512", "set_disk_normal", "rsqrt")])
def test_regions_of_the_path_tracers(name, label, op):
    k = ir.load(name)
    b = next(b for b in k.blocks if b.label == label)
    rows, member = E.Lowering(k).table_rows(b.instrs)
    cond, inside = E.guarded_region(b.instrs, k.liveness()[1][b.idx], set(rows) | set(member))
    assert op in {b.instrs[p].op for p in inside}
    assert not any(b.instrs[p].op == "tab" for p in inside)
