"""Lower a Loom kernel (text IR) to CUDA C++ for the B200 engines.

For every kernel the generator writes one translation unit that defines a
struct ``K`` with

* ``Regs``            the Loom register file as scalars (kept in CUDA
                      registers); Union registers (Loom src/common/union.hpp)
                      are stored as unsigned integers and bit-cast per view;
* ``run_burst<kProf>`` the whole program as a goto CFG that can be entered at
                      any block and stops after a budget of blocks: the
                      plain engine runs it from block 0 with the step guard
                      as budget, the regrouping engine runs bursts of a few
                      blocks between warp votes;
* ``save/restore(b)`` the live-in registers of block b to/from the queue of
                      block b (an SoA segment per block and round parity);
* ``load_inputs`` / ``store_outputs`` the input/output columns;

plus the host-side descriptor and launchers.  Op semantics follow Loom
src/vm/operators.hpp and the std:: functors exactly as standard_eval applies
them (core.hpp:740-750): arguments are converted to the functor's operand
type, the functor's result type is kept (T for arithmetic, bool for
comparisons and logic), and the result is converted to the destination
variable's type.  The TU is compiled with -fmad=false and IEEE division and
square root so that float arithmetic rounds like the scalar backend.
"""

from __future__ import annotations

import math
import struct
from typing import Dict, List

from .ir import (
    FLOAT_TYPES,
    HALT,
    INT_TYPES,
    TYPE_BYTES,
    Compute,
    Jump,
    Kernel,
    Operand,
    ParmJump,
)


# Register cap of the regrouping megakernel.  The persistent kernel keeps
# every lane busy from one resident warp set, so latency is hidden only by
# the warps an SM holds: 64 registers fit 2 CTAs of 512 threads (32 warps)
# per SM, against 16 warps at the compiler's own choice of 128 for the
# sphere path tracer.  The spills this costs stay in L1; measured on one
# B200, 1024x768x64 sphere path tracer 41.0 ms vs 52.5 ms, 256 batched
# render requests 156.6 ms vs 180.4 ms, outputs identical.
REGROUP_MAX_REGS = 64

# Further register caps compiled for kernels large enough to reach the cap
# (more static instructions than REG_VARIANT_MIN_INSTR): the tuner picks one
# per workload (opts.max_regs), trading warps per SM against spills.
REG_VARIANTS = (32, 40, 48, 56, 80, 96, 128)
REG_VARIANT_MIN_INSTR = 300
# Small kernels: the megakernel's own state dominates their registers, and a
# cap that fits one more CTA per SM can pay for latency-bound loops.
SMALL_REG_VARIANTS = (40, 48)

# Long blocks: at least this many instructions.  The software-stepped
# schedule can hold lanes that reach one back until enough of the warp's
# lanes stand there (opts.defer_lanes), so that its long code runs at a
# higher lane efficiency (the path tracers' random-number subroutine).
LONG_BLOCK_INSTR = 96


# Table reads of one block up to this many words above the lowest one of
# their record share its address (kFlatWords in engine/common.cuh leaves that
# much room below 2^32).  The path tracer's intersection loop is issue-bound
# and reads 4 words an iteration, which cost 3 instructions each with an
# index of their own: 48 batched render requests 19.87 -> 17.53 ms, 320x240x16
# with default options 3.38 -> 2.97 ms, the 1024x768x64 render 25.94 -> 25.22
# ms.  One 128-bit load behind a check of the alignment was slower than four
# words at constant offsets (lane-efficiency form 4.46 against 4.22 ms): the
# branch pins the loads in a block of their own.
ROW_SPAN = 63


def long_blocks(k: Kernel) -> List[int]:
    """Blocks of at least LONG_BLOCK_INSTR instructions, longest first (at
    most 4)."""
    counts = k.instr_counts()
    return sorted((b for b in range(k.num_blocks) if counts[b] >= LONG_BLOCK_INSTR), key=lambda b: -counts[b])[:4]


def any_order(k: Kernel) -> bool:
    """Whether schedule 2 needs no order among the blocks where lanes can
    stand (block 0 and those where a step may end): one loop at most, and no
    long block among several, for which lanes may have to wait."""
    steps = k.step_headers(set(long_blocks(k)))
    stands = steps | {0}
    return len(steps) <= 1 and (len(stands) == 1 or not stands & set(long_blocks(k)))


# Copies of a block that loops on itself: (most instructions, copies with an
# exit each, copies of a counted loop without).  A look at the iterations left, the loop's condition and its counter cost as
# much as a short body.  Copies with one look per group: 2^20 Fibonacci
# threads 48.5 -> 35.9 us.  Where the condition compares a counter with a
# bound, whole groups run without it (counted_loop): 19.5 us, and the path
# tracer's intersection loop, whose 38 instructions lose to the code size with
# exits in every copy (default options 2.47 -> 2.60 ms), gains with four plain
# ones (2.25 ms; 1024x768x64 render 23.7 -> 22.8 ms; 48 batched requests 15.9 ->
# 14.1 ms; two copies: 2.40, 22.9 and 14.1 ms).
UNROLL = ((12, 8, 8), (24, 4, 4), (48, 1, 4))


def unroll_factor(blk) -> int:
    """Copies of a block that loops on itself, by its instructions."""
    t = blk.terminator
    if not (isinstance(t, ParmJump) and len(t.targets) == 2 and not t.var.is_literal) or t.targets.count(blk.idx) != 1:
        return 1
    c = 2 if counted_loop(blk) else 1
    return next((u[c] for u in UNROLL if len(blk.instrs) <= u[0]), 1)


def counted_loop(blk):
    """(counter, bound, comparison) of a block that loops on itself while a
    counter it steps by one compares with a bound it does not change: `i + 1`
    written once, then compared, integers of 32 or 64 bits; else None."""
    t = blk.terminator
    if not isinstance(t, ParmJump) or t.var.is_literal or len(t.targets) != 2 or t.targets[1] != blk.idx:
        return None
    ins = blk.instrs[:-1]
    at = max((p for p, x in enumerate(ins) if x.dst.reg == t.var.reg), default=-1)
    if at < 0:
        return None
    c = ins[at]
    if c.op not in ("lt", "le", "ne", "gt", "ge") or c.optype[0] not in ("u32", "i32", "u64", "i64"):
        return None
    flip = {"lt": "gt", "le": "ge", "gt": "lt", "ge": "le", "ne": "ne"}
    for i, n, cmp in ((c.args[0], c.args[1], c.op), (c.args[1], c.args[0], flip[c.op])):
        if i.is_literal or cmp not in ("lt", "le", "ne") or i.type != c.optype[0] or n.type != c.optype[0]:
            continue
        steps = [p for p, x in enumerate(ins) if x.dst.reg == i.reg]
        if len(steps) != 1 or steps[0] > at or i.reg == t.var.reg:
            continue
        s = ins[steps[0]]
        one = [a for a in s.args if a.is_literal and a.value() == 1]
        if s.op != "add" or s.optype != c.optype or s.dst != i or len(one) != 1 or i not in s.args:
            continue
        if not n.is_literal and any(x.dst.reg == n.reg for x in ins):
            continue
        return i, n, cmp
    return None


def bit_heavy(blk) -> bool:
    """Whether a long block is mostly shifts and logic, which only the ALU pipe
    runs, at half the issue rate.  In programs without loops, of which the SM
    holds warps enough to hide latency, its 32-bit sums then go to the
    multiply pipe: 2e7 Threefry counters 130 -> 118 us.  In the path tracers,
    whose serial rounds wait on latency, the longer multiply-add lost: the
    1024x768x64 render 22.8 -> 23.7 ms."""
    n = sum(1 for x in blk.instrs if isinstance(x, Compute) and x.op in ("bxor", "bor", "band", "shl", "shr"))
    return len(blk.instrs) >= LONG_BLOCK_INSTR and 2 * n >= len(blk.instrs)


def reg_caps(k: Kernel) -> List[int]:
    """Register caps of the megakernel compiled for `k`, default first."""
    extra = REG_VARIANTS if sum(k.instr_counts()) > REG_VARIANT_MIN_INSTR else SMALL_REG_VARIANTS
    return [REGROUP_MAX_REGS] + [c for c in extra if c != REGROUP_MAX_REGS]


CTYPE = {
    "b8": "bool",
    "i8": "signed char",
    "u8": "unsigned char",
    "i16": "short",
    "u16": "unsigned short",
    "i32": "int",
    "u32": "unsigned int",
    "i64": "long long",
    "u64": "unsigned long long",
    "f32": "float",
    "f64": "double",
}

ABI_TYPE = {
    "b8": "LOOM_B200_B8",
    "i8": "LOOM_B200_I8",
    "u8": "LOOM_B200_U8",
    "i16": "LOOM_B200_I16",
    "u16": "LOOM_B200_U16",
    "i32": "LOOM_B200_I32",
    "u32": "LOOM_B200_U32",
    "i64": "LOOM_B200_I64",
    "u64": "LOOM_B200_U64",
    "f32": "LOOM_B200_F32",
    "f64": "LOOM_B200_F64",
}

CMP = {"eq": "==", "ne": "!=", "gt": ">", "lt": "<", "ge": ">=", "le": "<="}
ARITH = {"add": "+", "sub": "-", "mul": "*", "div": "/", "mod": "%"}
BITS = {"band": "&", "bor": "|", "bxor": "^", "shl": "<<", "shr": ">>"}
LOGIC = {"land": "&&", "lor": "||"}
UNARY_FN = {
    "round": "op_round",
    "ceil": "op_ceil",
    "floor": "op_floor",
    "trunc": "op_trunc",
    "sqrt": "op_sqrt",
    "sin": "op_sin",
    "cos": "op_cos",
    "rsqrt": "op_rsqrt",
}


def literal(op: Operand) -> str:
    """Exact C++ spelling of a literal's bit pattern."""
    t = op.type
    ct = CTYPE[t]
    if t == "f32":
        v = struct.unpack("<f", struct.pack("<I", op.bits & 0xFFFFFFFF))[0]
        if math.isfinite(v):
            return f"({v.hex()}f)"
        return f"__uint_as_float({op.bits & 0xFFFFFFFF:#x}u)"
    if t == "f64":
        v = struct.unpack("<d", struct.pack("<Q", op.bits))[0]
        if math.isfinite(v):
            return f"({v.hex()})"
        return f"__longlong_as_double({op.bits:#x}ll)"
    if t == "b8":
        return "true" if op.bits & 1 else "false"
    nbits = TYPE_BYTES[t] * 8
    bits = op.bits & ((1 << nbits) - 1)
    return f"(({ct}){bits:#x}ull)"


# Rough issue slots of operations that cost many (division and square root
# with IEEE rounding, their slow paths left out); every other one counts 1.
OP_COST = {"div": 10, "mod": 20, "sqrt": 9, "rsqrt": 18, "sin": 60, "cos": 60}

# A region that only a condition needs moves behind it from this cost on (the
# branch and the reconvergence after it take 3 to 4 instructions).  The path
# tracer's intersection loop is issue-bound, a ray misses most spheres of a
# random scene, and the root of its clamped discriminant, 0, takes the square
# root's slow path (29 cycles a warp instead of 14): behind `hit = det >= 0`
# 48 batched requests run 1.28x as fast (15.9 ms), the 1024x768x64 render 24.58
# -> 23.69 ms, the serving burst 1.08x as fast.
SINK_MIN_COST = 12


# Selects of 64-bit integers: instructions of the predicated arm, at most.
ARM_MAX = 4
PTX_OP = {"add": "add.u64", "sub": "sub.u64", "mul": "mul.lo.u64", "band": "and.b64", "bor": "or.b64", "bxor": "xor.b64"}


def predicated_ptx(arm):
    """PTX of the instructions of an arm under predicate p, the last one's
    result in %0, and the registers it reads in operand order (from %2); a
    product that only the next sum reads becomes a mad.  None: not of plain
    64-bit integer operations."""
    value: Dict[int, str] = {}  # register -> its operand or temporary
    regs: List[int] = []

    def operand(a):
        if a.is_literal:
            return f"{a.bits & 0xFFFFFFFFFFFFFFFF:#x}"
        if a.reg not in value:
            value[a.reg] = f"%{2 + len(regs)}"
            regs.append(a.reg)
        return value[a.reg]

    text = []
    skip = False
    for j, x in enumerate(arm):
        if x.op not in PTX_OP or x.optype[0] not in ("u64", "i64") or any(a.type != x.optype[0] for a in x.args + [x.dst]):
            return None
        if skip:
            skip = False
            continue
        nxt = arm[j + 1] if j + 1 < len(arm) else None
        fused = (
            x.op == "mul" and nxt is not None and nxt.op == "add"
            and [not a.is_literal and a.reg == x.dst.reg for a in nxt.args] == [True, False]
            and (nxt.dst.reg == x.dst.reg or not any(x.dst.reg in y.reads() for y in arm[j + 2 :]))
            and all(a.type == nxt.optype[0] for a in nxt.args + [nxt.dst]) and nxt.optype[0] in ("u64", "i64")
        )
        args = [operand(a) for a in x.args]
        last = x
        if fused:
            args.append(operand(nxt.args[1]))
            last, skip = nxt, True
        end = last is arm[-1]
        dst = "%0" if end else f"t{j}"
        text.append(f"@p {'mad.lo.u64' if fused else PTX_OP[x.op]} {dst}, {', '.join(args)};")
        value[last.dst.reg] = dst
    return " ".join(text), regs


def select_arms(instrs, live_out, storage, barred=frozenset()) -> Dict[int, tuple]:
    """Selects of 64-bit integers whose operands are computed for them alone:
    {position of the cmov: (positions of the arm that runs in line, positions
    of the arm predicated over its result, whether that is the second
    value)}.  A 64-bit select costs two instructions on the ALU pipe, which
    bounds integer loops; with one arm predicated there is none (Collatz, a
    warp's iteration with all lanes busy: 17.2 -> 13.2 cycles).  Positions in
    `barred` (members of constant rows, emitted as such) join no arm."""
    n = len(instrs)
    reach: Dict[int, int] = {}  # register -> position of its last definition
    uses: Dict[int, List[tuple]] = {}  # definition -> [(position, operand)]
    for p, ins in enumerate(instrs):
        if isinstance(ins, Compute):
            for i, a in enumerate(ins.args):
                if not a.is_literal and a.reg in reach:
                    uses.setdefault(reach[a.reg], []).append((p, i))
            reach[ins.dst.reg] = p
        else:
            for r in ins.reads():
                if r in reach:
                    uses.setdefault(reach[r], []).append((p, 0))
    kept = {reach[r] for r in live_out if r in reach}
    out: Dict[int, tuple] = {}
    taken = set()
    for q, sel in enumerate(instrs):
        if not isinstance(sel, Compute) or sel.op != "cmov" or sel.dst.type not in ("u64", "i64"):
            continue
        arms = []
        for side in (1, 2):
            arm: set = set()
            grown = True
            while grown:
                grown = False
                for p in range(q):
                    if p in arm or p in taken or p in kept or p in barred or not isinstance(instrs[p], Compute):
                        continue
                    if instrs[p].op in OP_COST or instrs[p].op in ("assert_fp", "tab", "cmov"):
                        continue
                    u = uses.get(p, [])
                    if u and all(x == (q, side) or x[0] in arm for x in u):
                        arm.add(p)
                        grown = True
            arms.append(sorted(arm))
        # the arm with the products is predicated (the multiply pipe is not
        # the ALU's), the other one runs in line
        muls = [sum(instrs[p].op == "mul" for p in arm) for arm in arms]
        pick = 0 if muls[0] >= muls[1] else 1
        both = arms[0] + arms[1]
        if not arms[pick] or len(arms[pick]) > ARM_MAX or predicated_ptx([instrs[p] for p in arms[pick]]) is None:
            continue
        if instrs[arms[pick][-1]].dst != sel.args[1 + pick] or any(not a.is_literal and a.type != sel.dst.type for a in sel.args[1:]):
            continue
        # they move down to the select: nothing in between may change what
        # they read, or touch what they write
        ok = all(storage[r] in ("u64", "i64") for p in arms[pick] for r in instrs[p].reads() + instrs[p].writes())
        for p in both:
            for m in range(p + 1, q):
                if m in both or not isinstance(instrs[m], Compute):
                    continue
                d = instrs[m].dst.reg
                if d in instrs[p].reads() or d == instrs[p].dst.reg:
                    ok = False
        regs = [{instrs[p].dst.reg for p in arm} for arm in arms]
        # ... and the arm in line, which runs first, nothing the other reads
        line = {instrs[p].dst.reg for p in arms[1 - pick]}
        ok = ok and not line & set(predicated_ptx([instrs[p] for p in arms[pick]])[1])
        if ok and not (sel.args[0].is_literal or sel.args[0].reg in regs[0] | regs[1]):
            out[q] = (arms[1 - pick], arms[pick], pick == 1)
            taken |= set(both) | {q}
    return out


def guarded_region(instrs, live_out, fixed, arms=None):
    """Work of a block that only matters while a condition register holds
    true: (position of the instruction that sets the register, positions of
    the work), or None.

    Loom kernels are written without branches: `hit = det >= 0`, then the
    root, the nearer of two distances, `hit = hit && t < tmin`, `tmin = hit ?
    t : tmin`.  With the register false, `r = r && x` leaves it false, a
    conditional move under it that keeps its own register does nothing, and
    what else feeds only those has no effect, so a lane whose condition is
    false may skip all of it.  The rest of the block (`fixed` positions are
    part of it, as are instructions with side effects) runs after the region,
    and only where that order gives the same values: order meaning that of the
    generated code, where the arms of a select (`arms`, from select_arms) stand
    right before it.  Of all conditions the one with the costliest region is
    taken."""
    best, best_cost = None, SINK_MIN_COST - 1
    n = len(instrs)
    last = n - 1 if n and not isinstance(instrs[-1], Compute) else n
    arms = arms or {}
    moved = {p for line, asm, _ in arms.values() for p in line + asm}
    # predicated: their results never reach their registers
    unwritten = {p for _, asm, _ in arms.values() for p in asm}
    order = []
    for p in range(last):
        if p in arms:
            order += arms[p][0] + arms[p][1]
        if p not in moved:
            order.append(p)
    for at, c in enumerate(order):
        h = instrs[c]
        if c in moved:
            continue
        after = order[at + 1 :]
        if h.op not in CMP and h.op not in LOGIC and h.op != "pacc":
            continue
        reg = h.dst.reg
        known = {reg}  # registers that hold false while the condition does
        noop = set()
        for q in after:
            ins = instrs[q]
            first = None if not ins.args or ins.args[0].is_literal else ins.args[0].reg
            same = first == ins.dst.reg
            if ins.op == "cmov" and first in known and ins.args[2] == ins.dst:
                noop.add(q)
            elif (
                (ins.op == "pacc" and ins.optype[2] == "land" or ins.op == "land")
                and first in known and same and ins.args[0] == ins.dst and ins.dst.type in INT_TYPES
            ):
                noop.add(q)
            elif ins.dst.reg in known:
                known.discard(ins.dst.reg)
                if not known:
                    break
        # backwards: what is read while the condition is false
        live = set(live_out) | ({r for r in instrs[-1].reads()} if last < n else set())
        skip = set()
        for q in reversed(after):
            ins = instrs[q]
            if q in noop and q not in fixed:
                skip.add(q)
            elif ins.dst.reg in live or q in fixed or ins.op == "assert_fp":
                if q not in unwritten:
                    live.discard(ins.dst.reg)
                live |= set(ins.reads())
            else:
                skip.add(q)
        # the region in order, then the rest: cut where the order matters
        inside = []
        rest = []
        for q in after:
            ins = instrs[q]
            if q not in skip:
                rest.append(q)
                continue
            if any(
                instrs[r].dst.reg in ins.reads() or instrs[r].dst.reg == ins.dst.reg or ins.dst.reg in instrs[r].reads()
                for r in rest
            ):
                # this one and all later ones stay where they are
                rest.append(q)
                continue
            inside.append(q)
        # what stays may not need, while the condition is false, a register
        # that the region would have set: true by liveness for the skipped
        # set as a whole, so a cut set is checked again
        if len(inside) != len(skip):
            live = set(live_out) | ({r for r in instrs[-1].reads()} if last < n else set())
            ok = True
            for q in reversed(after):
                ins = instrs[q]
                if q in inside:
                    if q not in noop and ins.dst.reg in live:
                        ok = False
                        break
                    continue
                if q not in unwritten:
                    live.discard(ins.dst.reg)
                live |= set(ins.reads())
            if not ok:
                continue
        cost = sum(OP_COST.get(instrs[q].op, 1) for q in inside)
        if cost > best_cost:
            best, best_cost = (c, set(inside)), cost
    return best


# Selections among constants by one index: from this many on they become
# 128-bit loads from one row of constant memory.  A chain of compares and
# selects costs some 4 ALU instructions per value and entry count of 5 (Loom's
# path tracers fetch a box side's 12 coordinates so on every test); lanes that
# traverse together read one row.  A 384x384 window of Loom's pt_const 53.9 ->
# 51.4 ms.
SCT_MIN = 3

# Bytes of a kernel's constant rows, at most: constant memory holds 65536, of
# which the engine's own tables take 8 a block.  The largest selections of
# Loom's path tracers take 560 bytes a kernel.  What does not fit stays a
# chain of selects.
SCT_BYTES = 48 << 10


class Lowering:
    def __init__(self, k: Kernel, device: bool = False):
        self.k = k
        self.pc = k.pc_reg()
        self.regs = {r.idx: r for r in k.regs}
        # expressions for device code (the CPU restatement of the gang engine
        # lowers with this class too, without the device's helpers)
        self.device = device
        self.mad_adds = False
        # (block, first position) of the constant rows that fit
        self.rows_kept = set()
        left = SCT_BYTES
        for b in k.blocks:
            for first, (_, n, ps) in self.constant_rows(b.instrs).items():
                size = n * ((len(ps) + 3) // 4) * 16
                if size <= left:
                    left -= size
                    self.rows_kept.add((b.idx, first))

    # ------------------------------------------------------------ views
    def rname(self, idx: int) -> str:
        return f"R.r{idx}"

    def read(self, op: Operand) -> str:
        if op.is_literal:
            return literal(op)
        reg = self.regs[op.reg]
        if reg.storage == op.type:
            return self.rname(op.reg)
        return f"bitcast<{CTYPE[op.type]}>({self.rname(op.reg)})"

    def write(self, dst: Operand, expr: str) -> str:
        reg = self.regs[dst.reg]
        val = f"static_cast<{CTYPE[dst.type]}>({expr})"
        if reg.storage == dst.type:
            return f"{self.rname(dst.reg)} = {val};"
        return f"{self.rname(dst.reg)} = bitcast<{CTYPE[reg.storage]}>({val});"

    # ------------------------------------------------------------ ops
    def expr(self, ins: Compute) -> str:
        op = ins.op
        a = [self.read(x) for x in ins.args]
        ot = ins.optype

        def cv(i: int, t: str) -> str:
            return f"static_cast<{CTYPE[t]}>({a[i]})"

        if op == "mov":
            return a[0]
        if op == "cmov":
            return f"(({a[0]}) ? ({a[1]}) : ({a[2]}))"
        if op in ("fma", "fms"):
            t = ins.args[0].type
            z = a[2] if op == "fma" else f"(-({a[2]}))"
            return f"op_fma({a[0]}, {a[1]}, {z})"
        if op == "assert_fp":
            return f"op_assert_fp({a[0]}, ctx)"
        if op == "tab":
            (t,) = ot
            return f"table_load<{CTYPE[t]}>(*ctx.cols, static_cast<unsigned>({a[0]}))"
        if op == "sct":
            t, _ = ot
            consts = [literal(c) for c in ins.consts]
            idx = a[0]
            e = consts[-1]
            for i in reversed(range(len(consts) - 1)):
                e = f"(({idx}) == {i} ? {consts[i]} : {e})"
            return f"static_cast<{CTYPE[t]}>({e})"
        if op == "slt":
            t, _ = ot
            idx = a[0]
            vals = a[1:]
            e = f"static_cast<{CTYPE[t]}>({vals[-1]})"
            for i in reversed(range(len(vals) - 1)):
                e = f"(({idx}) == {i} ? static_cast<{CTYPE[t]}>({vals[i]}) : {e})"
            return e
        if op == "pacc":
            t, it, acc, cmp = ot
            c = f"static_cast<{CTYPE[it]}>({cv(1, t)} {CMP[cmp]} {cv(2, t)})"
            return f"static_cast<{CTYPE[it]}>({cv(0, it)} {LOGIC[acc]} {c})"
        (t,) = ot
        ct = CTYPE[t]
        if op == "add" and t == "u32" and self.mad_adds:
            return f"op_add_mad({cv(0, t)}, {cv(1, t)}, ctx.cols->one)"
        if op in ARITH:
            return f"static_cast<{ct}>({cv(0, t)} {ARITH[op]} {cv(1, t)})"
        if op in BITS:
            return f"static_cast<{ct}>({cv(0, t)} {BITS[op]} {cv(1, t)})"
        if op in ("eq", "ne") and t in ("u64", "i64") and self.device:
            # against a literal below 2^32: one three-input logic operation
            # on the halves that sets the predicate, instead of a compare of
            # each half (the ALU pipe takes two cycles for either)
            for i, lit in ((0, ins.args[1]), (1, ins.args[0])):
                if lit.is_literal and lit.type in INT_TYPES and not ins.args[i].is_literal and lit.value() in range(1 << 32):
                    v = f"static_cast<{CTYPE['u64']}>({cv(i, t)})"
                    return f"{'' if op == 'ne' else '!'}op_differs({v}, {lit.value():#x}u)"
        if op in CMP:
            return f"static_cast<bool>({cv(0, t)} {CMP[op]} {cv(1, t)})"
        if op in LOGIC:
            return f"static_cast<bool>({cv(0, t)} {LOGIC[op]} {cv(1, t)})"
        if op == "lnot":
            return f"static_cast<bool>(!{cv(0, t)})"
        if op == "neg":
            return f"static_cast<{ct}>(-{cv(0, t)})"
        if op == "bnot":
            return f"static_cast<{ct}>(~{cv(0, t)})"
        if op == "abs":
            if t in FLOAT_TYPES:
                return f"op_abs({cv(0, t)})"
            if t.startswith("u"):
                return cv(0, t)
            wide = "long long" if t == "i64" else "int"
            return f"static_cast<{ct}>(op_abs(static_cast<{wide}>({cv(0, t)})))"
        if op == "max":
            return f"op_max<{ct}>({cv(0, t)}, {cv(1, t)})"
        if op == "min":
            return f"op_min<{ct}>({cv(0, t)}, {cv(1, t)})"
        if op == "copysign":
            return f"op_copysign({cv(0, t)}, {cv(1, t)})"
        if op in UNARY_FN:
            return f"{UNARY_FN[op]}({cv(0, t)})"
        raise NotImplementedError(f"{self.k.name}: op {op}")

    def table_rows(self, instrs):
        """Table reads of a block that stand at literal distances from one
        another (a record's fields): every index register is followed through
        moves and additions of literals, and the reads whose index comes from
        one value, at most ROW_SPAN words from the lowest, form a row.
        Returns {position of the row's first read: (index expression of the
        lowest read, [distances from it])} and {position of a read: (position
        of its row's first read, distance)}."""
        origin: Dict[int, tuple] = {}  # register -> (value, distance from it)
        values = 0
        reads: Dict[int, List[tuple]] = {}  # value -> [(position, distance)]
        for pos, ins in enumerate(instrs):
            if not isinstance(ins, Compute):
                continue
            for a in ins.args:
                if not a.is_literal and a.reg not in origin:
                    origin[a.reg] = (values, 0)
                    values += 1
            a = ins.args[0]
            if ins.op == "tab" and not a.is_literal and a.type == "u32":
                v, d = origin[a.reg]
                reads.setdefault(v, []).append((pos, d))
            new = (values, 0)
            if ins.dst.type == "u32" and ins.op == "mov" and not a.is_literal and a.type == "u32":
                new = origin[a.reg]
            elif ins.dst.type == "u32" and ins.op == "add" and ins.optype == ("u32",):
                for x, y in (ins.args, ins.args[::-1]):
                    if y.is_literal and not x.is_literal and x.type == "u32":
                        v, d = origin[x.reg]
                        new = (v, (d + y.bits) & 0xFFFFFFFF)
                        break
            if new[0] == values:
                values += 1
            origin[ins.dst.reg] = new
        rows: Dict[int, tuple] = {}
        member: Dict[int, tuple] = {}
        for r in reads.values():
            lo = min(d for _, d in r)
            r = [(p, d - lo) for p, d in r if d - lo <= ROW_SPAN]
            dist = sorted({d for _, d in r})
            if len(dist) < 2:
                continue
            first, d0 = r[0]
            base = self.read(instrs[first].args[0])
            rows[first] = (base if d0 == 0 else f"{base} - {d0}u", dist)
            for p, d in r:
                member[p] = (first, d)
        return rows, member

    def constant_rows(self, instrs, block=None):
        """Selections among constants (`sct`) by one index: {position of the
        first: (index operand, entries, positions)} of every SCT_MIN or more
        of them on an index that does not change in between, with the same
        number of 4-byte entries.  With the number of the block: those of
        them that constant memory has room for."""
        groups: Dict[tuple, List[int]] = {}
        version: Dict[int, int] = {}
        for p, ins in enumerate(instrs):
            if not isinstance(ins, Compute):
                continue
            a = ins.args[0] if ins.args else None
            if (
                ins.op == "sct" and not a.is_literal and a.type in ("u8", "u16", "u32", "u64")
                and len(ins.consts) >= 3 and all(TYPE_BYTES[c.type] == 4 for c in ins.consts)
            ):
                groups.setdefault((a.reg, version.get(a.reg, 0), len(ins.consts)), []).append(p)
            version[ins.dst.reg] = version.get(ins.dst.reg, 0) + 1
        rows = {ps[0]: (instrs[ps[0]].args[0], n, ps) for (_, _, n), ps in groups.items() if len(ps) >= SCT_MIN}
        return {p: r for p, r in rows.items() if block is None or (block, p) in self.rows_kept}

    def constant_tables(self, blk) -> List[str]:
        """Definitions of a block's constant rows: an entry's values side by
        side, padded to whole 16-byte words."""
        out = []
        for first, (_, n, ps) in self.constant_rows(blk.instrs, blk.idx).items():
            rows = []
            for i in range(n):
                words = [f"{blk.instrs[p].consts[i].bits & 0xFFFFFFFF:#x}u" for p in ps]
                words += ["0u"] * (-len(words) % 4)
                rows += ["{" + ", ".join(words[j : j + 4]) + "}" for j in range(0, len(words), 4)]
            out.append(f"__constant__ uint4 kSct{blk.idx}_{first}[{len(rows)}] = {{{', '.join(rows)}}};")
        return out

    def body(self, instrs, indent: str, live_out=None, block: int = 0) -> List[str]:
        """The instructions of a block (without its terminator).  `live_out`:
        registers read after them, which allows work that only a condition
        needs to move behind it."""
        rows, member = self.table_rows(instrs)

        sct = self.constant_rows(instrs, block)
        sct_of = {p: (first, j) for first, (_, _, ps) in sct.items() for j, p in enumerate(ps)}

        def emit(pos: int, indent: str) -> List[str]:
            out = []
            ins = instrs[pos]
            if pos in sct:
                idx, n, ps = sct[pos]
                width = (len(ps) + 3) // 4
                # 8 and 16 bits need not hold the last entry's number
                ct = CTYPE["u64" if idx.type == "u64" else "u32"]
                out.append(indent + f"const uint4* sp{pos} = kSct{block}_{pos} + {width}u * static_cast<unsigned>(op_min<{ct}>({self.read(idx)}, {n - 1}));")
                out.extend(indent + f"const uint4 sv{pos}_{j} = sp{pos}[{j}];" for j in range(width))
            if pos in sct_of:
                first, j = sct_of[pos]
                (t, _) = ins.optype
                out.append(indent + self.write(ins.dst, f"bitcast<{CTYPE[t]}>(sv{first}_{j // 4}.{'xyzw'[j % 4]})"))
                return out
            if pos in arms:
                # one arm in line, the other predicated over its result
                line, asm, inverted = arms[pos]
                for p in line:
                    out.append(indent + self.write(instrs[p].dst, self.expr(instrs[p])))
                ct = CTYPE[ins.dst.type]
                c = f"static_cast<unsigned>(static_cast<bool>({self.read(ins.args[0])}))"
                out.append(indent + "{")
                out.append(indent + f"    unsigned long long v = static_cast<unsigned long long>({self.read(ins.args[1 if inverted else 2])});")
                text, regs = predicated_ptx([instrs[p] for p in asm])
                ops = ", ".join([f'"r"({c})'] + [f'"l"({self.rname(r)})' for r in regs])
                out.append(indent + f'    asm("{{.reg .pred p; .reg .u64 t<{len(asm) + 1}>; setp.{"eq" if inverted else "ne"}.u32 p, %1, 0; {text}}}"')
                out.append(indent + f'        : "+l"(v) : {ops});')
                out.append(indent + "    " + self.write(ins.dst, f"static_cast<{ct}>(v)"))
                out.append(indent + "}")
                return out
            if pos in rows:
                base, dist = rows[pos]
                out.append(indent + f"const unsigned tb{pos} = static_cast<unsigned>({base});")
                out.append(indent + "if constexpr(kFlat)")
                out.append(indent + "{")
                out.append(indent + f"    const unsigned* tp = ctx.cols->table + tb{pos};")
                out.extend(indent + f"    tw{pos}_{d} = __ldg(tp + {d});" for d in dist)
                out.append(indent + "}")
                out.append(indent + "else")
                out.append(indent + "{")
                out.extend(indent + f"    tw{pos}_{d} = table_load<unsigned>(*ctx.cols, tb{pos} + {d}u);" for d in dist)
                out.append(indent + "}")
            if pos in member:
                first, d = member[pos]
                (t,) = ins.optype
                out.append(indent + self.write(ins.dst, f"bitcast<{CTYPE[t]}>(tw{first}_{d})"))
            else:
                out.append(indent + self.write(ins.dst, self.expr(ins)))
            return out

        todo = [p for p, ins in enumerate(instrs) if isinstance(ins, Compute)]
        storage = {i: r.storage for i, r in self.regs.items()}
        arms = select_arms(instrs, live_out, storage, sct_of) if live_out is not None else {}
        in_arm = {p for a, b, _ in arms.values() for p in a + b}
        todo = [p for p in todo if p not in in_arm]
        out = []
        inner = indent + "    " if rows or sct else indent
        for pos in rows:
            out.append(inner + f"unsigned {', '.join(f'tw{pos}_{d}' for d in rows[pos][1])};")
        fixed = set(rows) | set(member) | set(sct_of) | set(arms) | in_arm
        sink = guarded_region(instrs, live_out, fixed, arms) if live_out is not None else None
        if sink:
            cond, inside = sink
            for p in todo:
                if p <= cond:
                    out.extend(emit(p, inner))
            out.append(inner + f"if({self.read(instrs[cond].dst)})")
            out.append(inner + "{")
            for p in todo:
                if p in inside:
                    out.extend(emit(p, inner + "    "))
            out.append(inner + "}")
            todo = [p for p in todo if p > cond and p not in inside]
        for p in todo:
            out.extend(emit(p, inner))
        if rows or sct:  # a scope of their own: labels of other blocks are jumped to past them
            out = [indent + "{"] + out + [indent + "}"]
        return out

    # ------------------------------------------------------------ transfers
    def next_expr(self, blk) -> str:
        """C++ expression of the next block index (kHalt for HALT)."""
        t = blk.terminator
        if t is None:
            return "kHalt"
        if isinstance(t, Jump):
            return self.target(t.target)
        v = self.read(t.var)
        tg = [self.target(x) for x in t.targets]
        if len(tg) == 2:
            # Loom's scalar dispatch: any non-zero selects the second label
            # (bse.hpp:180-185).
            return f"(({v}) ? {tg[1]} : {tg[0]})"
        e = "kHalt"  # out-of-table values leave the thread where it is
        for i in reversed(range(len(tg))):
            e = f"(({v}) == {i} ? {tg[i]} : {e})"
        return e

    @staticmethod
    def target(t: int) -> str:
        return "kHalt" if t == HALT else str(t)

    def goto_transfer(self, blk, indent: str) -> List[str]:
        t = blk.terminator
        if t is None:
            return [indent + "goto L_HALT;"]
        if isinstance(t, Jump):
            return [indent + f"goto {self.label(t.target)};"]
        v = self.read(t.var)
        if len(t.targets) == 2:
            return [
                indent
                + f"if({v}) goto {self.label(t.targets[1])}; else goto {self.label(t.targets[0])};"
            ]
        lines = [indent + f"switch({v}) {{"]
        for i, tg in enumerate(t.targets):
            lines.append(indent + f"case {i}: goto {self.label(tg)};")
        lines.append(indent + "default: goto L_HALT;")
        lines.append(indent + "}")
        return lines

    @staticmethod
    def label(t: int) -> str:
        return "L_HALT" if t == HALT else f"L_B{t}"


def pack_slots(items, start: int) -> Dict:
    """Queue row layout from `start` (bytes per entry): items (register,
    bytes) and the input index ("tid", 4).  Registers of 8 and 4 bytes and
    the index are packed largest first into slots of 16 bytes, each at an
    offset that is a multiple of its size; the last slot shrinks to 8 or 4
    bytes when that holds its contents; registers of 1 or 2 bytes get a slot
    each.  Returns {"slots": [(off, width, [(item, sub)])], "cols": {reg: (off,
    sub, width)}, "tid": (off, sub, width), "end": next offset, a multiple
    of 8}."""
    wide = sorted([(r, n) for r, n in items if n >= 4], key=lambda x: (-x[1], x[0])) + [("tid", 4)]
    narrow = sorted([(r, n) for r, n in items if n < 4], key=lambda x: (-x[1], x[0]))
    slots = []
    cur, used = [], 0
    for it, n in wide:
        if used + n > 16:
            slots.append((cur, used))
            cur, used = [], 0
        cur.append((it, used, n))
        used += n
    if cur:
        slots.append((cur, used))
    out, off = [], start
    for contents, used in slots:
        width = 16 if used > 8 else (8 if used > 4 else 4)
        out.append((off, width, [(it, sub) for it, sub, _ in contents]))
        off += width
    for it, n in narrow:
        out.append((off, n, [(it, 0)]))
        off += n
    end = (off + 7) // 8 * 8
    cols, tid = {}, None
    for o, wdt, contents in out:
        for it, sub in contents:
            if it == "tid":
                tid = (o, sub, wdt)
            else:
                cols[it] = (o, sub, wdt)
    return {"slots": out, "cols": cols, "tid": tid, "end": end}


def generate(k: Kernel) -> str:
    L = Lowering(k, device=True)
    name = k.name
    nb = k.num_blocks
    nin = len(k.inputs)
    nout = len(k.outputs)
    live_in, live_outs = k.liveness()
    state = k.state_regs()
    counts = k.instr_counts()
    live_bytes = [sum(L.regs[r].nbytes for r in li) for li in live_in]
    regs = [r for r in k.regs if r.idx != L.pc]
    if nin + nout > 96:
        raise ValueError(f"{name}: too many columns")
    # work queues: one per block plus one per context of each dispatch block
    queues = k.queues()
    qlive = k.queue_liveness()
    disp = k.dispatch_blocks()
    nq = len(queues)
    qbytes = [sum(L.regs[r].nbytes for r in li) for li in qlive]
    # queue segments: per queue, the live-in registers and the u32 input
    # index packed into slots of 16 bytes per entry (then 8, 4: the rest),
    # so a lane saves or restores four 32-bit values with one 128-bit access
    # and a warp's 32 entries of a slot are 512 contiguous bytes; registers
    # of 1 or 2 bytes keep slots of their own
    layout = []
    row_total = 0
    for q in range(nq):
        layout.append(pack_slots([(r, L.regs[r].nbytes) for r in qlive[q]], row_total))
        row_total = layout[-1]["end"]

    o: List[str] = []
    w = o.append
    w(f"// Generated by loom_b200.codegen from loom_b200/ir/{name}.lir.")
    w(f"// Kernel IR digest {k.digest()}; regenerate instead of editing.")
    w('#include "../engine/plain.cuh"')
    w('#include "../engine/regroup.cuh"')
    w('#include "../runtime_iface.h"')
    w("")
    w(f"namespace loom_b200 {{ namespace k_{name} {{")
    w("")
    w(f"__constant__ unsigned kInstrTab[{nb}] = {{{', '.join(map(str, counts))}}};")
    w(f"__constant__ unsigned kLiveTab[{nq}] = {{{', '.join(map(str, qbytes))}}};")
    w(f"__constant__ int kQueueBlock[{nq}] = {{{', '.join(str(b) for b, _ in queues)}}};")
    # Regrouping cost model: a group of g lanes at block b either runs it
    # now (I_b warp instructions) or parks (C_b column stores now, C_b loads
    # per restored tile of 32, then I_b at full width); parking is cheaper
    # while g < 32 (I_b - C_b) / (I_b + C_b), which is the block's quorum.
    quorum = []
    for b in range(nb):
        cols = max((len(qlive[q]) for q, (qb, _) in enumerate(queues) if qb == b), default=0) + 1
        ib = counts[b]
        quorum.append(min(28, max(0, math.ceil(32 * (ib - cols) / (ib + cols)))) if ib > cols else 0)
    heavy = {b for b in range(nb) if quorum[b] > 0}
    w(f"__constant__ unsigned kQuorumTab[{nb}] = {{{', '.join(map(str, quorum))}}};")
    w(f"__constant__ unsigned kRankTab[{nb}] = {{{', '.join(map(str, k.rpo_ranks()))}}};")
    for blk in k.blocks:
        o.extend(L.constant_tables(blk))
    w("")
    w("struct K")
    w("{")
    w(f"    static constexpr int kNumBlocks = {nb};")
    w(f"    static constexpr int kNumQueues = {nq};")
    w(f"    static constexpr int kRegroupMaxRegs = {REGROUP_MAX_REGS};")
    # small kernels: two inlined copies of their code in the megakernel
    w(f"    static constexpr bool kSplitCallSites = {'true' if sum(counts) <= REG_VARIANT_MIN_INSTR else 'false'};")
    w(f"    static constexpr bool kAnyOrder = {str(any_order(k)).lower()}; // schedule 2: lanes need no order")
    spread = bool(k.loop_headers()) and sum(counts) > REG_VARIANT_MIN_INSTR
    w(f"    static constexpr bool kSpread = {str(spread).lower()}; // a large program with loops")
    # kernels that read records of the table: their launches on flat tables
    # run instantiations of their own
    table_rows = any(L.table_rows(b.instrs)[0] for b in k.blocks)
    w(f"    static constexpr bool kTableRows = {'true' if table_rows else 'false'};")
    w("    struct Regs")
    w("    {")
    for r in regs:
        w(f"        {CTYPE[r.storage]} r{r.idx}; // {r.name}: {','.join(r.types)}")
    if not regs:
        w("        int unused;")
    w("    };")
    w("")
    # ---- inputs / outputs
    w("    struct In")
    w("    {")
    for i, (reg, t, vname) in enumerate(k.inputs):
        w(f"        {CTYPE[t]} v{i}; // {vname}")
    if not k.inputs:
        w("        int unused;")
    w("    };")
    w("")
    w("    // Reads the input columns of thread `tid` (a NULL column is iota).")
    w("    __device__ __forceinline__ static void")
    w("    load_in(In& in, const Columns& c, const unsigned long long tid)")
    w("    {")
    for i, (reg, t, vname) in enumerate(k.inputs):
        w(f"        in.v{i} = load_input<{CTYPE[t]}>(c, {i}, tid);")
    w("        (void)in; (void)c; (void)tid;")
    w("    }")
    w("")
    w("    // Loom's set_inputs: input variables written, every other register zero.")
    w("    // Only registers live at START (those its queue carries) are written:")
    w("    // the others are written before they are read on every path.")
    w("    __device__ __forceinline__ static void")
    w("    start(Regs& R, const In& in)")
    w("    {")
    live0 = qlive[queues.index((0, None))] if k.blocks else set()
    in_regs = {reg for reg, _, _ in k.inputs}
    for r in regs:
        if r.idx in live0 and r.idx not in in_regs:
            w(f"        R.r{r.idx} = 0;")
    for i, (reg, t, vname) in enumerate(k.inputs):
        w("        " + L.write(Operand(type=t, reg=reg), f"in.v{i}"))
    w("        (void)in;")
    w("    }")
    w("")
    w("    __device__ __forceinline__ static void")
    w("    load_inputs(Regs& R, const Columns& c, const unsigned long long tid)")
    w("    {")
    w("        In in;")
    w("        load_in(in, c, tid);")
    w("        start(R, in);")
    w("    }")
    w("")
    w("    __device__ __forceinline__ static void")
    w("    store_outputs(const Regs& R, const Columns& c, const unsigned long long tid)")
    w("    {")
    for j, (reg, t, vname) in enumerate(k.outputs):
        ct = CTYPE[t]
        w(f"        static_cast<{ct}*>(c.p[{nin + j}])[col_index(c, tid)] = {L.read(Operand(type=t, reg=reg))}; // {vname}")
    w("    }")
    w("")
    w("    __device__ __forceinline__ static unsigned instr(const int b) { return kInstrTab[b]; }")
    w("    __device__ __forceinline__ static unsigned live_bytes(const int q) { return kLiveTab[q]; }")
    w("    __device__ __forceinline__ static int block_of(const int q) { return kQueueBlock[q]; }")
    w("    __device__ __forceinline__ static unsigned quorum(const int b) { return kQuorumTab[b]; }")
    w("    __device__ __forceinline__ static unsigned rank(const int b) { return kRankTab[b]; }")
    lb = long_blocks(k)
    w(f"    static constexpr int kNumLong = {len(lb)};")
    w("    // j-th long block (most instructions first)")
    w("    __device__ __forceinline__ static int long_block(const int j)")
    w("    {")
    if lb:
        w("        switch(j)")
        w("        {")
        for j, b in enumerate(lb):
            w(f"        case {j}: return {b};")
        w("        default: return -1;")
        w("        }")
    else:
        w("        (void)j;")
        w("        return -1;")
    w("    }")
    w("")
    per_block = [[qi for qi, (b, _) in enumerate(queues) if b == blk] for blk in range(nb)]
    maxq = max(len(x) for x in per_block)
    w(f"    static constexpr int kMaxQueuesPerBlock = {maxq};")
    w("    // j-th queue holding threads that stand at block b (-1: none).")
    w("    __device__ __forceinline__ static int")
    w("    queue_list(const int b, const int j)")
    w("    {")
    multi = [(blk, ql) for blk, ql in enumerate(per_block) if len(ql) > 1]
    for blk, ql in multi:
        w(f"        if(b == {blk})")
        w("        {")
        w("            switch(j)")
        w("            {")
        for j, qi in enumerate(ql):
            w(f"            case {j}: return {qi};")
        w("            default: return -1;")
        w("            }")
        w("        }")
    w("        return j == 0 ? b : -1;")
    w("    }")
    w("")
    w("    // Queue a thread standing at block pc waits in: the block's own queue,")
    w("    // or for a dispatch block the queue of the context its register selects.")
    w("    __device__ __forceinline__ static int")
    w("    queue_of(const int pc, const Regs& R)")
    w("    {")
    w("        (void)R;")
    for d, (v, ctx) in sorted(disp.items()):
        w(f"        if(pc == {d})")
        w("        {")
        w(f"            switch(static_cast<unsigned long long>(R.r{v}))")
        w("            {")
        for kk in ctx:
            w(f"            case {kk}ull: return {queues.index((d, kk))};")
        w("            default: break;")
        w("            }")
        w("        }")
    w("        return pc;")
    w("    }")
    w("")
    # ---- run_burst (goto CFG entered at any block, bounded by a budget)
    # the budget is counted at loop headers only (targets of edges that go
    # back in reverse post-order): every cycle passes one, and the blocks in
    # between have no early exit, so a diverged warp reconverges at their
    # post-dominators as in straight CUDA
    headers = k.loop_headers()
    # the regrouping engine's steps end at a minimal set of headers that
    # every cycle passes: a step costs it some 30 instructions, and the path
    # tracer's `bounce`, which runs into the intersection loop's own header,
    # only added steps (1024x768x64 render 25.2 -> 24.6 ms without it); the
    # long blocks stay, where lanes may have to wait for others.  The plain
    # engine spends its step guard at every header.
    steps = k.step_headers(set(long_blocks(k)))
    w("    // Runs the lane's own path from block `entry` for at most `budget`")
    w("    // loop iterations (visits of a loop header); returns the block it")
    w("    // stopped at, or kHalt.  With `stop_heavy`, a block whose quorum is")
    w("    // above zero is entered only as the first block of the burst, when")
    w("    // the warp's vote chose it.  A block that loops on itself takes up")
    w("    // to `spin` iterations (not 0) for one of the budget (a loop the")
    w("    // warp's lanes run together needs no step of its own per iteration).")
    w("    // kFlat: the launch's table is flat (Columns::table_flat).  kAllHeaders:")
    w("    // every loop header spends budget (the plain engine's step guard);")
    w("    // otherwise a minimal set of them that every cycle passes.")
    w("    template <bool kProf, bool kFlat, bool kAllHeaders>")
    w("    __device__ __forceinline__ static int")
    w("    run_burst(const int entry, Regs& R, Ctx& ctx, const unsigned budget, const bool stop_heavy = false,")
    w("              unsigned spin = 0u)")
    w("    {")
    w("        return run_steps<kProf, kFlat, kAllHeaders>(entry, R, ctx, budget, stop_heavy, spin);")
    w("    }")
    w("    // ... which takes the iterations it ran off `spin` (programs of several")
    w("    // loops; one loop's last iterations stay uncounted, as only HALT follows).")
    w("    template <bool kProf, bool kFlat, bool kAllHeaders>")
    w("    __device__ __forceinline__ static int")
    w("    run_steps(const int entry, Regs& R, Ctx& ctx, unsigned budget, const bool stop_heavy, unsigned& spin)")
    w("    {")
    w("        (void)ctx;")
    w("        (void)stop_heavy;")
    w("        (void)spin;")
    if any(unroll_factor(b) > 1 for b in k.blocks):
        w("        unsigned left = 0u; // iterations of a self-loop left")
        w("        unsigned sure = 0u; // of them, those that surely go on")
        w("        (void)sure;")
    w("        bool fresh = true; // no block run yet in this burst")
    w("        (void)fresh;")
    w("        switch(entry)")
    w("        {")
    for blk in k.blocks:
        w(f"        case {blk.idx}: goto L_B{blk.idx};")
    w("        default: return kHalt;")
    w("        }")
    for blk in k.blocks:
        b = blk.idx
        w(f"    L_B{b}: // {blk.label}")
        transfer = L.goto_transfer(blk, "        ")
        own = f"goto L_B{b};"
        self_loop = b in headers and b in blk.successors()
        copies = unroll_factor(blk) if self_loop else 1
        if b in heavy or self_loop:
            # a lane that loops on the block keeps going; one that comes
            # from another block waits for the warp's vote
            if b in heavy:
                w(f"        if(stop_heavy && !fresh) return {b};")
            w(f"    L_B{b}_again:")
        body = []
        if heavy:
            body.append("        fresh = false;")
        body.append(f"        if constexpr(kProf) count_block(ctx, {b}, {len(blk.instrs)}u);")
        L.mad_adds = not headers and bit_heavy(blk)
        body.extend(L.body(blk.instrs, "        ", live_outs[b], b))
        if copies > 1:
            # iterations until the budget has to be looked at again, run in
            # groups of `copies` with one look at their number per group
            stay = f"({L.read(blk.terminator.var)})"
            if blk.terminator.targets[0] == b:
                stay = f"!{stay}"
            other = next(t for t in blk.terminator.targets if t != b)
            # a loop that only HALT can follow leaves the counters alone (the
            # ordered form of programs of several loops reads them)
            ends = not (k.reachable(other) & headers) and len(steps) <= 1
            counted = counted_loop(blk)
            w(f"        if(budget == 0u) return {b};")
            w("        left = spin ? spin : budget;")
            if counted:
                # iterations after which the loop surely goes on need no
                # look at its condition
                i, n, cmp = counted
                w(f"        sure = loop_more_{cmp}<{CTYPE[i.type]}>({L.read(i)}, {L.read(n)}, left);")
                w("        left -= sure;")
                u = copies
                while u > 1:
                    w(f"        {'while' if u == copies else 'if'}(sure >= {u}u)")
                    w("        {")
                    for j in range(u):
                        o.extend("    " + ln for ln in body)
                    w(f"            sure -= {u}u;")
                    w("        }")
                    u //= 2
                w("        left += sure;")
            else:
                w(f"        while(left >= {copies}u)")
                w("        {")
                for j in range(1, copies + 1):
                    o.extend("    " + ln for ln in body)
                    if ends:
                        w(f"            if(!{stay}) goto {L.label(other)};")
                    else:
                        w(f"            if(!{stay}) {{ left -= {j}u; goto L_B{b}_out; }}")
                w(f"            left -= {copies}u;")
                w("        }")
            w("        while(left)")
            w("        {")
            o.extend("    " + ln for ln in body)
            w("            --left;")
            w(f"            if(!{stay}) goto {L.label(other) if ends else f'L_B{b}_out'};")
            w("        }")
            w("        if(spin) { spin = 0u; --budget; } else budget = 0u;")
            w(f"        goto L_B{b}_again;")
            if not ends:
                w(f"    L_B{b}_out:")
                w("        if(spin) { spin = left; --budget; } else budget = left;")
                w(f"        goto {L.label(other)};")
            continue
        if self_loop:
            back = f"{{ if(spin != 0u) {{ --spin; goto L_B{b}_spin; }} goto L_B{b}_again; }}"
            transfer = [t.replace(own, back) for t in transfer]
        elif b in heavy:
            transfer = [t.replace(own, f"goto L_B{b}_again;") for t in transfer]
        if b in steps:
            w(f"        if(budget == 0u) return {b};")
            w("        --budget;")
            if self_loop:
                w("        if(spin) --spin;")
        elif b in headers:
            w(f"        if(kAllHeaders && budget == 0u) return {b};")
            w("        if(kAllHeaders) --budget;")
        if self_loop:
            w(f"    L_B{b}_spin:")
        o.extend(body)
        o.extend(transfer)
    w("    L_HALT:")
    w("        return kHalt;")
    w("    }")
    w("")
    # ---- save / restore: queue (parity, block) holds the block's live-in
    # registers and the input index, one SoA column each
    w(f"    static constexpr unsigned long long kRowBytes = {row_total}ull;")
    for fn in ("save", "restore"):
        w("    __device__ __forceinline__ static " + ("void" if fn == "save" else "unsigned"))
        if fn == "save":
            w("    save(const int q, const Regs& R, char* st, const unsigned cap, const unsigned par,")
            w("         const unsigned idx, const unsigned tid)")
        else:
            w("    restore(const int q, Regs& R, const char* st, const unsigned cap, const unsigned par,")
            w("            const unsigned idx)")
        w("    {")
        q = "" if fn == "save" else "const "
        w(f"        {q}char* base = st + static_cast<unsigned long long>(par) * kRowBytes * cap;")
        w("        switch(q)")
        w("        {")
        for qi, (b, kk) in enumerate(queues):
            w(f"        case {qi}: // {k.blocks[b].label}" + ("" if kk is None else f", context {kk}"))
            w("        {")
            if fn == "restore" and kk is not None:
                v = disp[b][0]
                w(f"            R.r{v} = static_cast<{CTYPE[L.regs[v].storage]}>({kk});")
            tid_expr = None
            for si, (off, wdt, contents) in enumerate(layout[qi]["slots"]):
                vt = {16: "uint4", 8: "uint2", 4: "unsigned", 2: "unsigned short", 1: "unsigned char"}[wdt]
                slot = f"reinterpret_cast<{q}{vt}*>(base + {off}ull * cap)[idx]"
                if wdt <= 2:
                    # a narrow register alone in its slot
                    (r, _), = contents
                    stt = CTYPE[L.regs[r].storage]
                    if fn == "save":
                        w(f"            {slot} = bitcast<{vt}>(R.r{r});")
                    else:
                        w(f"            R.r{r} = bitcast<{stt}>({slot});")
                    continue
                words = ["x", "y", "z", "w"][: wdt // 4] if wdt > 4 else [None]
                def word(sub):
                    return f"v{si}" if words == [None] else f"v{si}.{words[sub // 4]}"
                if fn == "save":
                    w(f"            {{")
                    w(f"                {vt} v{si};")
                    for it, sub in contents:
                        if it == "tid":
                            w(f"                {word(sub)} = tid;")
                        elif L.regs[it].nbytes == 8:
                            w(f"                {{ const unsigned long long b = bitcast<unsigned long long>(R.r{it});")
                            w(f"                  {word(sub)} = static_cast<unsigned>(b); {word(sub + 4)} = static_cast<unsigned>(b >> 32); }}")
                        else:
                            w(f"                {word(sub)} = bitcast<unsigned>(R.r{it});")
                    w(f"                {slot} = v{si};")
                    w(f"            }}")
                else:
                    w(f"            const {vt} v{si} = {slot};")
                    for it, sub in contents:
                        if it == "tid":
                            tid_expr = word(sub)
                        elif L.regs[it].nbytes == 8:
                            stt = CTYPE[L.regs[it].storage]
                            w(f"            R.r{it} = bitcast<{stt}>((static_cast<unsigned long long>({word(sub + 4)}) << 32) | {word(sub)});")
                        else:
                            stt = CTYPE[L.regs[it].storage]
                            w(f"            R.r{it} = bitcast<{stt}>({word(sub)});")
            if fn == "save":
                w("            return;")
            else:
                w(f"            return {tid_expr};")
            w("        }")
        w("        default: " + ("return;" if fn == "save" else "return 0xffffffffu;"))
        w("        }")
        w("    }")
        w("")
    # ---- bulk-copy restore: a tile's 32 entries of every slot column are 32
    # consecutive slots, so one cp.async.bulk per slot column brings the
    # tile into shared memory, where each lane reads its own entries
    stage_rows = []
    for qi in range(nq):
        stage_rows.append(sum(wdt for _, wdt, _ in layout[qi]["slots"]))
    max_stage = max(stage_rows) if stage_rows else 16
    max_stage = (max_stage + 15) // 16 * 16
    w("    // bytes of one queue entry's slots, the largest over the queues")
    w(f"    static constexpr unsigned kMaxStageRow = {max_stage}u;")
    w("    // Lane 0 of a warp: copies the full tile [toff, toff + 32) of queue q")
    w("    // (state half `base`) into `stage` (32 x kMaxStageRow bytes of shared")
    w("    // memory) with one bulk copy per slot column, completing on the")
    w("    // mbarrier at `mbar`; false (nothing issued) when an address is not on")
    w("    // a 16-byte boundary.")
    w("    __device__ __forceinline__ static bool")
    w("    bulk_issue(const int q, unsigned char* stage, const char* base, const unsigned cap, const unsigned toff,")
    w("               unsigned long long* mbar)")
    w("    {")
    w("        unsigned bytes = 0;")
    w("        switch(q)")
    w("        {")
    for qi in range(nq):
        w(f"        case {qi}: bytes = {32 * stage_rows[qi]}u; break;")
    w("        default: return false;")
    w("        }")
    w("        if((reinterpret_cast<unsigned long long>(base) | reinterpret_cast<unsigned long long>(stage)) & 15ull) return false;")
    w("        bulk_expect(mbar, bytes);")
    w("        switch(q)")
    w("        {")
    for qi in range(nq):
        w(f"        case {qi}:")
        so = 0
        for off, wdt, _ in layout[qi]["slots"]:
            w(f"            bulk_copy(stage + {so}u, base + {off}ull * cap + static_cast<unsigned long long>(toff) * {wdt}u, {32 * wdt}u, mbar);")
            so += 32 * wdt
        w("            break;")
    w("        default: break;")
    w("        }")
    w("        return true;")
    w("    }")
    w("")
    w("    // A lane's entry of a tile staged by bulk_issue; returns its thread id.")
    w("    __device__ __forceinline__ static unsigned")
    w("    restore_stage(const int q, Regs& R, const unsigned char* stage, const unsigned lane)")
    w("    {")
    w("        switch(q)")
    w("        {")
    for qi, (b, kk) in enumerate(queues):
        w(f"        case {qi}:")
        w("        {")
        if kk is not None:
            v = disp[b][0]
            w(f"            R.r{v} = static_cast<{CTYPE[L.regs[v].storage]}>({kk});")
        tid_expr = None
        so = 0
        for si, (off, wdt, contents) in enumerate(layout[qi]["slots"]):
            vt = {16: "uint4", 8: "uint2", 4: "unsigned", 2: "unsigned short", 1: "unsigned char"}[wdt]
            slot = f"reinterpret_cast<const {vt}*>(stage + {so}u)[lane]"
            so += 32 * wdt
            if wdt <= 2:
                (r, _), = contents
                w(f"            R.r{r} = bitcast<{CTYPE[L.regs[r].storage]}>({slot});")
                continue
            words = ["x", "y", "z", "w"][: wdt // 4] if wdt > 4 else [None]

            def word(sub, si=si, words=words):
                return f"v{si}" if words == [None] else f"v{si}.{words[sub // 4]}"

            w(f"            const {vt} v{si} = {slot};")
            for it, sub in contents:
                if it == "tid":
                    tid_expr = word(sub)
                elif L.regs[it].nbytes == 8:
                    w(f"            R.r{it} = bitcast<{CTYPE[L.regs[it].storage]}>((static_cast<unsigned long long>({word(sub + 4)}) << 32) | {word(sub)});")
                else:
                    w(f"            R.r{it} = bitcast<{CTYPE[L.regs[it].storage]}>({word(sub)});")
        w(f"            return {tid_expr};")
        w("        }")
    w("        default: return 0xffffffffu;")
    w("        }")
    w("    }")
    w("};")
    w("")
    # ---- host side
    w("const int kInTypes[] = {" + ", ".join(ABI_TYPE[t] for _, t, _ in k.inputs) + "};")
    w("const int kOutTypes[] = {" + ", ".join(ABI_TYPE[t] for _, t, _ in k.outputs) + "};")
    w("const char* const kInNames[] = {" + ", ".join(f'"{n}"' for _, _, n in k.inputs) + "};")
    w("const char* const kOutNames[] = {" + ", ".join(f'"{n}"' for _, _, n in k.outputs) + "};")
    w(f"const uint32_t kInstrs[] = {{{', '.join(map(str, counts))}}};")
    w(f"const uint32_t kLive[] = {{{', '.join(map(str, live_bytes))}}};")
    state_size = sum(r.nbytes for r in k.regs)
    w("")
    w("const loom_b200_kernel_info kInfo = {")
    w(f'    "{name}", "{k.digest()}", {nin}u, {nout}u, kInTypes, kOutTypes, kInNames, kOutNames,')
    w(f"    {nb}u, {len(k.regs)}u, {state_size}u, {len(state)}u, kInstrs, kLive}};")
    w("")
    # queue layouts for state inspection: the block (and dispatch context)
    # of each queue, its columns in save order and where they lie in a row
    assert all(rg.idx == i for i, rg in enumerate(k.regs)), "registers out of order"
    assert all(qk is None or -(2**31) <= qk < 2**31 for _, qk in queues), "dispatch context out of range"
    for qi, (qb, qk) in enumerate(queues):
        # columns in register-size order (the order of the queue analysis)
        cols = sorted(layout[qi]["cols"], key=lambda r: (-L.regs[r].nbytes, r))
        layout[qi]["order"] = cols
        if cols:
            at = layout[qi]["cols"]
            w(f"const uint32_t kQRegs{qi}[] = {{{', '.join(f'{r}u' for r in cols)}}};")
            w(f"const int kQTypes{qi}[] = {{{', '.join(ABI_TYPE[L.regs[r].storage] for r in cols)}}};")
            names = ", ".join('"' + k.regs[r].name + '"' for r in cols)
            w(f"const char* const kQNames{qi}[] = {{{names}}};")
            w(f"const unsigned long long kQOffs{qi}[] = {{{', '.join(f'{at[r][0]}ull' for r in cols)}}};")
            w(f"const unsigned kQSubs{qi}[] = {{{', '.join(f'{at[r][1]}u' for r in cols)}}};")
            w(f"const unsigned kQWidths{qi}[] = {{{', '.join(f'{at[r][2]}u' for r in cols)}}};")
    w("const loom_b200_queue_layout kQueues[] = {")
    for qi, (qb, qk) in enumerate(queues):
        cols = layout[qi]["order"]
        if cols:
            w(f"    {{{qb}u, {-1 if qk is None else qk}, {len(cols)}u, kQRegs{qi}, kQTypes{qi}, kQNames{qi}}},")
        else:
            w(f"    {{{qb}u, {-1 if qk is None else qk}, 0u, nullptr, nullptr, nullptr}},")
    w("};")
    w("const QueueSegment kSegments[] = {")
    for qi in range(nq):
        has = bool(layout[qi]["order"])
        offs = f"kQOffs{qi}, kQSubs{qi}, kQWidths{qi}" if has else "nullptr, nullptr, nullptr"
        t = layout[qi]["tid"]
        w(f"    {{{offs}, {t[0]}ull, {t[1]}u, {t[2]}u}},")
    w("};")
    w("")
    flat = "true" if table_rows else "false"
    w("const void* plain_fn(bool profile, bool flat, unsigned per)")
    w("{")
    w("    if(profile) return reinterpret_cast<const void*>(&plain_kernel<K, true, false, 1>);")
    if table_rows:
        w("    if(!flat) return reinterpret_cast<const void*>(&plain_kernel<K, false, false, 1>);")
    several = not k.loop_headers() and not table_rows
    if not several:
        w("    (void)per;")
    else:
        w(f"    if(per > 1u) return reinterpret_cast<const void*>(&plain_kernel<K, false, {flat}, kStraightPer>);")
    w("    (void)flat;")
    w(f"    return reinterpret_cast<const void*>(&plain_kernel<K, false, {flat}, 1>);")
    w("}")
    w("")
    w("cudaError_t launch_plain(const PlainLaunch& a)")
    w("{")
    w("    const bool               flat = a.cols.table_flat != 0u;")
    w("    const unsigned long long cta  = a.lanes < 32u ? a.lanes : static_cast<unsigned long long>(a.block) * a.per;")
    w("    const unsigned long long grid = (a.n + cta - 1) / cta;")
    w("    if(grid == 0) return cudaSuccess;")
    w("    const void* fn     = plain_fn(a.profile, flat, a.per);")
    w("    void*       args[] = {const_cast<Columns*>(&a.cols), const_cast<unsigned long long*>(&a.first),")
    w("                          const_cast<unsigned long long*>(&a.n), const_cast<unsigned long long*>(&a.max_steps),")
    w("                          const_cast<unsigned**>(&a.status), const_cast<unsigned long long**>(&a.counters),")
    w("                          const_cast<unsigned*>(&a.lanes)};")
    w("    return cudaLaunchKernel(fn, dim3(static_cast<unsigned>(grid)), dim3(a.block), args, 0, a.stream);")
    w("}")
    w("")
    w("// registers of a thread of the plain kernel, and the threads a CTA of it can have")
    w("cudaError_t plain_attrs(bool profile, bool flat, unsigned per, int* regs, int* max_threads)")
    w("{")
    w("    cudaFuncAttributes  at{};")
    w("    const cudaError_t e = cudaFuncGetAttributes(&at, plain_fn(profile, flat, per));")
    w("    *regs        = at.numRegs;")
    w("    *max_threads = at.maxThreadsPerBlock;")
    w("    return e;")
    w("}")
    w("")
    caps = reg_caps(k)
    w(f"const unsigned kRegCaps[] = {{{', '.join(f'{c}u' for c in caps)}}};")
    w("")
    w("/// The megakernel at register cap `regs` (0: the default), in its form")
    w("/// for launches of `form`; profiled launches")
    w("/// and launches with the staged restore (`bulk`) use the default cap and")
    w("/// the parking form, and so do launches of a kernel with table records on")
    w("/// a table that is not flat (the staged-restore instantiation reads")
    w("/// every word by its own index).  NULL: no such cap compiled.")
    w("const void* regroup_fn(unsigned regs, bool profile, bool bulk, RegroupForm form, bool flat)")
    w("{")
    ordered = len(k.step_headers(set(long_blocks(k)))) > 1
    if ordered:
        w("    const bool ordered = form == RegroupForm::kParkOrdered && (regs == 0u || regs == K::kRegroupMaxRegs) && !bulk && flat;")
        w("    if(profile && ordered) return reinterpret_cast<const void*>(&regroup_kernel<K, true, K::kRegroupMaxRegs, false, true, true>);")
    w("    if(profile) return reinterpret_cast<const void*>(&regroup_kernel<K, true, K::kRegroupMaxRegs, true>);")
    w("    if(bulk) return reinterpret_cast<const void*>(&regroup_kernel<K, false, K::kRegroupMaxRegs, true>);")
    w("    if(K::kTableRows && !flat)")
    w("    {")
    w("        bool known = regs == 0u;")
    w("        for(const unsigned c: kRegCaps) known |= c == regs;")
    w("        return known ? reinterpret_cast<const void*>(&regroup_kernel<K, false, K::kRegroupMaxRegs, true>) : nullptr;")
    w("    }")
    w("    const bool park = form != RegroupForm::kNeverPark;")
    if ordered:
        w("    if(ordered) return reinterpret_cast<const void*>(&regroup_kernel<K, false, K::kRegroupMaxRegs, false, true, true>);")
    w("    switch(regs)")
    w("    {")
    w("    case 0u:")
    for c in caps:
        w(f"    case {c}u: return park ? reinterpret_cast<const void*>(&regroup_kernel<K, false, {c}, false, true>)")
        w(f"                          : reinterpret_cast<const void*>(&regroup_kernel<K, false, {c}, false, false>);")
    w("    default: return nullptr;")
    w("    }")
    w("}")
    w("")
    w("cudaError_t launch_regroup(const RegroupLaunch& a)")
    w("{")
    w("    void* args[] = {const_cast<RegroupParams*>(&a.params)};")
    w("    const void* fn = regroup_fn(a.regs, a.profile, a.params.bulk_restore != 0u, a.form, a.params.cols.table_flat != 0u);")
    w("    if(!fn) return cudaErrorInvalidValue;")
    w("    if(a.dyn_smem)")
    w("    {")
    w("        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,")
    w("                                                   static_cast<int>(a.dyn_smem));")
    w("        if(e != cudaSuccess) return e;")
    w("    }")
    w("    if(a.ordinary && a.params.slice_rounds == 1u)")
    w("        return cudaLaunchKernel(fn, dim3(a.grid), dim3(a.block), args, a.dyn_smem, a.stream);")
    w("    return cudaLaunchCooperativeKernel(fn, dim3(a.grid), dim3(a.block), args, a.dyn_smem, a.stream);")
    w("}")
    w("")
    w("cudaError_t regroup_occupancy(int block, bool profile, unsigned regs, unsigned dyn_smem, RegroupForm form, bool flat,")
    w("                              int* ctas)")
    w("{")
    w("    const void* fn = regroup_fn(regs, profile, dyn_smem != 0u, form, flat);")
    w("    if(!fn) return cudaErrorInvalidValue;")
    w("    if(dyn_smem)")
    w("    {")
    w("        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,")
    w("                                                   static_cast<int>(dyn_smem));")
    w("        if(e != cudaSuccess) return e;")
    w("    }")
    w("    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fn, block, dyn_smem);")
    w("}")
    w("")
    w(f"}} }} // namespace loom_b200::k_{name}")
    w("")
    w(f"extern const loom_b200::KernelEntry loom_b200_entry_{name};")
    w(f"const loom_b200::KernelEntry loom_b200_entry_{name} = {{")
    w(f"    &loom_b200::k_{name}::kInfo, loom_b200::k_{name}::K::kRowBytes, {nq},")
    w(f"    &loom_b200::k_{name}::launch_plain, &loom_b200::k_{name}::launch_regroup,")
    w(f"    &loom_b200::k_{name}::regroup_occupancy,")
    w(f"    &loom_b200::k_{name}::plain_attrs,")
    w(f"    loom_b200::k_{name}::kQueues, loom_b200::k_{name}::kSegments,")
    w(f"    loom_b200::k_{name}::kRegCaps, {len(caps)}u, loom_b200::k_{name}::K::kMaxStageRow, loom_b200::k_{name}::K::kSpread, {"loom_b200::kStraightPer" if several else "1u"}}};")
    return "\n".join(o) + "\n"


def generate_registry(names: List[str]) -> str:
    o = ["// Generated by loom_b200.codegen: the kernels compiled into libloom_b200.", ""]
    o.append('#include "../runtime_iface.h"')
    o.append("")
    for n in names:
        o.append(f"extern const loom_b200::KernelEntry loom_b200_entry_{n};")
    o.append("")
    o.append("namespace loom_b200 {")
    o.append("const KernelEntry* const kRegistry[] = {")
    for n in names:
        o.append(f"    &loom_b200_entry_{n},")
    o.append("};")
    o.append(f"const int kRegistrySize = {len(names)};")
    o.append("} // namespace loom_b200")
    return "\n".join(o) + "\n"
