"""The C restatement under several threads of one process: parsing keeps no
state that another parse can see, and the timed CPU leg, which runs slices of
the threads in a pool, gives what one run gives.  Each body runs in a child
process, which a data race would abort (CPU)."""

import pathlib
import subprocess
import sys
import textwrap

ROOT = pathlib.Path(__file__).resolve().parents[1]


def _child(body: str) -> None:
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(body)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_programs_parse_in_several_threads_at_once():
    _child(
        """
        import concurrent.futures
        from oracle import oracle as O

        O.build_interp()
        O.Interp("fib_u64")
        names = ["sphere_pt_f32", "threefry_u32", "collatz_u64", "no op"] * 16

        def load(name):
            if name == "no op":
                try:
                    O.Interp(name, "loomir 1\\nreg 0 a 4 u32\\nblock 0 start 1\\ni nothing u32 r0:u32 r0:u32\\n")
                except ValueError as e:
                    return "unknown op nothing" in str(e)
                return False
            O.Interp(name)
            return True

        with concurrent.futures.ThreadPoolExecutor(16) as ex:
            assert all(ex.map(load, names))
        """
    )


def test_slices_of_the_cpu_leg_equal_one_run():
    _child(
        """
        import numpy as np
        import bench
        from loom_b200 import scenes as S
        from oracle import oracle as O

        O.ref_available = lambda: False
        run, kind, cores = bench._reference_runner()
        assert kind == "port"
        table, _ = S.pack([S.cornell_request(16, 16, 2, seed=9)])
        for n in (1, 2, 33, 257):
            ins = [np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32)]
            got = run("sphere_pt_f32", ins, table)
            want = O.Interp("sphere_pt_f32").run(ins, table=table)
            assert len(got) == len(want) and all(g.tobytes() == w.tobytes() for g, w in zip(got, want))
        """
    )


def test_slices_continue_the_thread_index():
    """A column that is left out holds the thread index."""
    _child(
        """
        import numpy as np
        import bench
        from oracle import oracle as O

        O.ref_available = lambda: False
        run, _, _ = bench._reference_runner()
        for name in ("bit_xor_u16", "bit_or_u64", "minmax_f32"):
            x = np.arange(300, 0, -1).astype(O.NP_TYPE[O.Interp(name).inputs[0][1]])
            got = run(name, [x, None], None)
            want = O.Interp(name).run([x, None], n=len(x))
            assert all(g.tobytes() == w.tobytes() for g, w in zip(got, want)), name
        """
    )
