"""Blocks as the generator emits them, all its rules together: random blocks
in which the arms of selects, work behind a condition and selections among
constants meet, compiled for the CPU in the emitted order and in program
order, leave the same live values (CPU)."""

import ctypes
import random
import re
import subprocess

import numpy as np
import pytest

from loom_b200.codegen import emit_cuda as E
from loom_b200.codegen import ir

# registers 0-3: u64, 4-7: u32, 8-11: f32
TYPES = ["u64"] * 4 + ["u32"] * 4 + ["f32"] * 4
SIZE = {"u64": 8, "u32": 4, "f32": 4}
HEAD = "loomir 1\nkernel t\nindex u32\nstraight 1\n" + "".join(f"reg {i} x{i} {SIZE[t]} {t}\n" for i, t in enumerate(TYPES))

PRELUDE = r"""
#include <cmath>
#include <cstring>
template <typename To, typename From> static To bitcast(From v) { static_assert(sizeof(To) == sizeof(From)); To r; memcpy(&r, &v, sizeof r); return r; }
template <typename T> static T op_min(T a, T b) { return b < a ? b : a; }
static float op_sqrt(float v) { return std::sqrt(v); }
static bool op_differs(unsigned long long v, unsigned lit) { return v != lit; }
#define __constant__ static const
struct uint4 { unsigned x, y, z, w; };
struct Regs { unsigned long long r0, r1, r2, r3; unsigned r4, r5, r6, r7; float r8, r9, r10, r11; };
"""

PTX = {"add.u64": "+", "sub.u64": "-", "mul.lo.u64": "*", "and.b64": "&", "or.b64": "|", "xor.b64": "^"}


def _host(lines):
    """The emitted lines with each inline-assembly statement as C++."""
    out = []
    it = iter(lines)
    for ln in it:
        if "asm(" not in ln:
            out.append(ln)
            continue
        args = next(it)
        sense, text = re.search(r"setp\.(eq|ne)\.u32 p, %1, 0; (.*)}\"", ln).groups()
        cond = re.search(r'"r"\((.*?)\)(?:, "l"|\);)', args).group(1)
        regs = re.findall(r'"l"\((R\.r\d+)\)', args)
        at = {"%0": "v", **{f"%{2 + i}": f"a{i}" for i in range(len(regs))}}
        out.append("{ " + " ".join(f"const unsigned long long a{i} = {r};" for i, r in enumerate(regs)))
        out.append(f"if(({cond}) {'==' if sense == 'eq' else '!='} 0u) {{ unsigned long long t0, t1, t2, t3, t4; (void)t0; (void)t1; (void)t2; (void)t3; (void)t4;")
        for op in re.findall(r"@p ([^;]*);", text):
            name, rest = op.split(" ", 1)
            d, *a = [at.get(x.strip(), x.strip() + ("ull" if x.strip().startswith("0x") else "")) for x in rest.split(",")]
            out.append(f"{d} = {a[0]} * {a[1]} + {a[2]};" if name == "mad.lo.u64" else f"{d} = {a[0]} {PTX[name]} {a[1]};")
        out.append("} }")
    return out


def _reg(rng, t):
    lo = TYPES.index(t)
    return f"r{rng.randrange(lo, lo + 4)}:{t}"


def _operand(rng, t):
    if t != "f32" and rng.random() < 0.15:
        return f"k{t}:{rng.choice([0, 1, 2, 3]):#x}"
    return _reg(rng, t)


def _line(rng, constants):
    u, f, w = (lambda t=t: _operand(rng, t) for t in ("u32", "f32", "u64"))
    kind = rng.choice(["w", "w", "sel", "cmp", "cmp", "land", "f", "f", "root", "fsel", "fsel", "wsel"] + ["sct"] * (2 * constants))
    if kind == "w":
        return f"i {rng.choice(['mul', 'mul', 'add', 'sub', 'bxor'])} u64 {_reg(rng, 'u64')} {w()} {w()}"
    if kind == "sel":
        return f"i cmov - {_reg(rng, 'u64')} {u()} {w()} {w()}"
    if kind == "cmp":
        return f"i {rng.choice(['gt', 'lt'])} f32 {_reg(rng, 'u32')} {f()} {f()}"
    if kind == "land":
        d = _reg(rng, "u32")
        return f"i pacc f32,u32,land,lt {d} {d} {f()} {f()}"
    if kind == "f":
        return f"i {rng.choice(['add', 'mul', 'div', 'div'])} f32 {_reg(rng, 'f32')} {f()} {f()}"
    if kind == "root":
        return f"i sqrt f32 {_reg(rng, 'f32')} {f()}"
    if kind == "fsel":
        d = _reg(rng, "f32")
        return f"i cmov - {d} {u()} {f()} {d}"
    if kind == "wsel":
        d = _reg(rng, "u64")
        return f"i cmov - {d} {u()} {w()} {d}"
    t = rng.choice(["f32", "u32"])
    return f"i sct {t},u32 {_reg(rng, t)} r4:u32 | " + " ".join(f"k{t}:{rng.choice([0, 1, 5, 0x3f800000, 0x40400000]):#x}" for _ in range(3))


def _block(rng, constants):
    """Lines of a block: random ones, and between some of them the form in
    which the rules meet: an arm, a condition, the arm's select, then work
    under the condition that may write what the arm reads."""
    out = [_line(rng, constants) for _ in range(rng.randint(0, 6))]
    if rng.random() < 0.8:
        t, a, b, s = (_reg(rng, "u64") for _ in range(4))
        h, g = _reg(rng, "u32"), _operand(rng, "u32")
        x, y, z = (_reg(rng, "f32") for _ in range(3))
        form = [f"i {rng.choice(['mul', 'add'])} u64 {t} {a} {b}", f"i lt f32 {h} {x} {y}",
                f"i cmov - {s} {g} {t} {a}" if rng.random() < 0.5 else f"i cmov - {s} {g} {a} {t}",
                f"i sqrt f32 {z} {x}", f"i div f32 {z} {z} {y}", f"i cmov - {y} {h} {z} {y}", f"i cmov - {b} {h} {a} {b}"]
        for ln in form:
            out.append(ln)
            if rng.random() < 0.15:
                out.append(_line(rng, constants))
    if constants and rng.random() < 0.5:
        # a row of three selections, one of which may feed one arm alone
        sct = [f"i sct u32,u32 r{r}:u32 r4:u32 | ku32:0x1 ku32:{rng.randrange(9):#x} ku32:0x3" for r in (5, 6, 7)]
        t, a, b, s = (_reg(rng, "u64") for _ in range(4))
        rng.shuffle(sct)
        out += sct + [f"i mov - {t} r{rng.choice([5, 6, 7])}:u32", f"i mul u64 {a} {a} {b}", f"i cmov - {s} r4:u32 {t} {a}"]
    return out + [_line(rng, constants) for _ in range(rng.randint(0, 4))]


@pytest.mark.parametrize("constants", [False, True])
def test_emitted_order_of_random_blocks(constants, tmp_path):
    rng = random.Random(23 + constants)
    src, lives, both = [PRELUDE], [], 0
    for n in range(700):
        lines = _block(rng, constants)
        live = sorted(rng.sample(range(12), rng.randint(2, 5)))
        k = ir.parse(HEAD + f"output {live[0]} {TYPES[live[0]]} o\nblock 0 START {len(lines)}\n" + "\n".join(lines) + "\nend\n")
        k.blocks[0].idx = n  # the constants' names
        L = E.Lowering(k, device=True)
        ins = k.blocks[0].instrs
        arms = E.select_arms(ins, set(live), dict(enumerate(TYPES)))
        emitted = _host(L.body(ins, "", set(live), n))
        both += bool(arms) and any(re.match(r"\s*if\(R\.", ln) for ln in emitted)
        src += L.constant_tables(k.blocks[0])
        src += [f'extern "C" void want{n}(Regs& R) {{', *(L.write(i.dst, L.expr(i)) for i in ins), "}"]
        src += [f'extern "C" void got{n}(Regs& R) {{', *emitted, "}"]
        lives.append((live, lines))
    (tmp_path / "b.cpp").write_text("\n".join(src))
    so = tmp_path / "b.so"
    r = subprocess.run(["g++", "-std=c++17", "-O0", "-w", "-ffp-contract=off", "-shared", "-fPIC", "-o", so, tmp_path / "b.cpp"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:2000]
    lib = ctypes.CDLL(str(so))
    rng = np.random.default_rng(5)
    fields = np.dtype([(f"r{i}", {"u64": "u8", "u32": "u4", "f32": "f4"}[t]) for i, t in enumerate(TYPES)], align=True)
    for n, (live, lines) in enumerate(lives):
        for _ in range(8):
            v = np.zeros(1, fields)
            for i, t in enumerate(TYPES):
                v[f"r{i}"] = rng.choice([-1.0, 0.5, 2.0, 9.0]) if t == "f32" else rng.choice([0, 1, 2, 7]) if t == "u32" else rng.integers(0, 1 << 40)
            want, got = v.copy(), v.copy()
            getattr(lib, f"want{n}")(ctypes.c_void_p(want.ctypes.data))
            getattr(lib, f"got{n}")(ctypes.c_void_p(got.ctypes.data))
            for i in live:
                a, b = want[f"r{i}"], got[f"r{i}"]
                assert a.tobytes() == b.tobytes() or (a != a and b != b), (n, i, v, a, b, lines)
    assert both > 60


@pytest.mark.parametrize("t", ["u8", "u16", "u32", "u64"])
@pytest.mark.parametrize("entries", [3, 256, 257, 300])
def test_index_types_of_constant_rows(t, entries, tmp_path):
    """Every index value takes its own entry, those from the last on the last,
    also where the index's type does not hold the number of entries."""
    n = ir.TYPE_BYTES[t]
    head = f"loomir 1\nkernel t\nindex u32\nstraight 1\nreg 0 i {n} {t}\n" + "".join(f"reg {r} x{r} 4 u32\n" for r in (1, 2, 3))
    lines = [f"i sct u32,{t} r{r}:u32 r0:{t} | " + " ".join(f"ku32:{e * 4 + r:#x}" for e in range(entries)) for r in (1, 2, 3)]
    k = ir.parse(head + f"input 0 {t} i\noutput 1 u32 x1\nblock 0 START 3\n" + "\n".join(lines) + "\nend\n")
    L = E.Lowering(k, device=True)
    b = k.blocks[0]
    assert len(L.constant_rows(b.instrs)) == 1
    ct = {1: "unsigned char", 2: "unsigned short", 4: "unsigned", 8: "unsigned long long"}[n]
    code = PRELUDE.replace("struct Regs", "struct Unused") + "\n".join(L.constant_tables(b)) + f"\nstruct Regs {{ {ct} r0; unsigned r1, r2, r3; }};\n"
    code += f'extern "C" void run({ct} i, unsigned* o) {{ Regs R{{i, 0, 0, 0}};\n' + "\n".join(L.body(b.instrs, "", {1, 2, 3}, 0)) + "\no[0] = R.r1; o[1] = R.r2; o[2] = R.r3; }"
    (tmp_path / "c.cpp").write_text(code)
    r = subprocess.run(["g++", "-std=c++17", "-O0", "-w", "-shared", "-fPIC", "-o", tmp_path / "c.so", tmp_path / "c.cpp"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[:2000]
    lib = ctypes.CDLL(str(tmp_path / "c.so"))
    arg = {1: ctypes.c_uint8, 2: ctypes.c_uint16, 4: ctypes.c_uint32, 8: ctypes.c_uint64}[n]
    out = (ctypes.c_uint32 * 3)()
    for i in sorted({0, 1, 2, 43, 44, 45, 127, 254, 255, 256, 257, 299, 300, 65535, 1 << 31, (1 << 32) + 1, (1 << 64) - 1}):
        if i >> (8 * n):
            continue
        lib.run(arg(i), out)
        assert list(out) == [min(i, entries - 1) * 4 + r for r in (1, 2, 3)], i


def _wide(entries, groups):
    """A kernel of `groups` blocks of four selections of `entries` each."""
    blocks = [f"block {b} b{b} 5\n" + "".join(f"i sct u32,u32 r{r}:u32 r0:u32 | " + " ".join(f"ku32:{e * b + r:#x}" for e in range(entries)) + "\n"
              for r in (1, 2, 3, 4)) + f"j {b + 1 if b + 1 < groups else -1}\n" for b in range(groups)]
    head = "loomir 1\nkernel t\nindex u32\nstraight 0\n" + "".join(f"reg {r} x{r} 4 u32\n" for r in range(5))
    return ir.parse(head + "input 0 u32 x0\noutput 1 u32 x1\n" + "".join(blocks) + "end\n")


@pytest.mark.parametrize("entries,groups,kept", [(3, 2, [0, 1]), (3072, 1, [0]), (3073, 1, []), (1024, 4, [0, 1, 2]), (2000, 2, [0]), (12000, 2, [])])
def test_constant_rows_that_fit_constant_memory(entries, groups, kept):
    """Rows beyond the kernel's share of constant memory stay selects."""
    k = _wide(entries, groups)
    L = E.Lowering(k, device=True)
    tables = [t for b in k.blocks for t in L.constant_tables(b)]
    assert [int(re.search(r"kSct(\d+)_0\[", t).group(1)) for t in tables] == kept
    assert sum(16 * int(re.search(r"\[(\d+)\]", t).group(1)) for t in tables) <= 49152
    for b in k.blocks:
        body = "\n".join(L.body(b.instrs, "", {1, 2, 3, 4}, b.idx))
        assert ("kSct" in body) == (b.idx in kept) and (" ? " in body) == (b.idx not in kept)
