"""What the library launches and allocates, on the CPU: a child process with
fake_cudart.c in place of the CUDA runtime, which runs no kernel but refuses what the real
one refuses (launch sizes, shared memory without the opt-in, a full device)."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
NOMEM, CUDA_ERROR, STATE = 2, 3, 6


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """run(code, **environment) -> (what the child printed, [(device, kernel, status,
    dynamic shared memory, opt-in) of every launch])"""
    if shutil.which("gcc") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("needs gcc and the CUDA headers")
    where = tmp_path_factory.mktemp("fake")
    so = str(where / "fake_cudart.so")
    subprocess.run(["gcc", "-O1", "-Wall", "-Werror", "-fPIC", "-shared", "-I" + os.path.join(CUDA, "include"),
                    os.path.join(HERE, "fake_cudart.c"), "-o", so], check=True)

    def child(code, **env):
        log = str(where / "log")
        open(log, "w").close()
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code)],
                           env=dict(os.environ, LD_PRELOAD=so, FAKE_CUDA_LOG=log, PYTHONPATH=ROOT,
                                    **{k: str(v) for k, v in env.items()}),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-3000:]
        with open(log) as f:
            rows = [line.split() for line in f]
        return r.stdout.split(), [(int(r[0]), r[1], *map(int, r[2:])) for r in rows]

    return child


PRELUDE = """
import ctypes as C, sys
import numpy as np, disccofan_gb300 as dcf
fail_in = C.c_int.in_dll(C.CDLL(None), "fake_fail_in")
memory, in_use = (C.c_size_t.in_dll(C.CDLL(None), "fake_" + n) for n in ("memory", "in_use"))
def status(f):
    try:
        f()
    except dcf.DcfError as e:
        return e.status
    return 0
"""


@pytest.mark.parametrize("least", [1, 1 << 40])
@pytest.mark.parametrize("shape,dtype,conn,rule", [((200, 230), "uint16", 8, "subtractive"), ((60, 70), "uint8", 4, "min"),
                                                   ((20, 30, 40), "float32", 6, "direct"), ((60, 70), "uint8", 4, "max")])
def test_nothing_is_launched_after_a_failed_launch(run, shape, dtype, conn, rule, least):
    """Whichever launch of a call fails, it is the call's last, and the call reports it."""
    said, rows = run(f"""
        img = np.zeros({shape}, np.{dtype})
        for k in range(1000):
            ctx = dcf.Context(0)
            fail_in.value = k
            made = []
            calls = [lambda: made.append(ctx.build(img, connectivity={conn}, tree_type="max", attribute=0)),
                     lambda: made[0].set_attribute(14), lambda: made[0].filter(14, 2.0, "{rule}"),
                     lambda: made[0].check(14), lambda: made[0].pattern_spectrum(14, np.float32([0, 1, 2]))]
            for call in calls:
                st = status(call)
                if st:
                    assert st == {CUDA_ERROR} and ctx.launches == k, (k, st, ctx.launches)
                    break
            else:
                break
        print(k)
        """, DCF_BASIN_MIN=least)
    assert int(said[0]) > 10
    assert sum(s != 0 for _, _, s, *_ in rows) == int(said[0])


def test_launches_of_a_batch_stop_at_a_failed_one(run):
    for least in (1, 1 << 40):
        said, rows = run(f"""
            shapes = [(40, 50), (70, 33)]
            pix = np.zeros(40 * 50 + 70 * 33, np.float32)
            lv = np.float32([0, 1, 2])
            for k in range(1000):
                ctx = dcf.Context(0)
                b = ctx.batch(shapes, np.float32, connectivity=8, attribute=13)
                fail_in.value = k
                st = status(lambda: b.run(pix, filter_attr=0, lam=3.0, spectrum=(13, lv, 0, lv), use_graph=False))
                b.close()
                if not st:
                    break
                assert st == {CUDA_ERROR} and ctx.launches == k, (k, st, ctx.launches)
            print(k)
            """, DCF_BASIN_MIN=least)
        assert int(said[0]) > 10
        assert sum(s != 0 for _, _, s, *_ in rows) == int(said[0])


@pytest.mark.parametrize("least", [1, 1 << 40])
def test_records_of_a_failed_attribute_pass_are_not_kept(run, least):
    """After a set_attribute that failed, whichever launch of it did, the tree has no
    attributes, and the next one computes them."""
    said, _ = run(f"""
        ctx = dcf.Context(0)
        t = ctx.build(np.zeros((50, 60), np.uint16), connectivity=8, tree_type="max", attribute=0)
        out = np.zeros(3000, np.float32)
        use = lambda: ctx.lib.dcf_filter(ctx.h, t.h, 14, 0, 2.0, 0, out.ctypes.data, 0)
        before = ctx.launches
        t.set_attribute(14)
        whole = ctx.launches - before
        t.set_attribute(0)
        for k in range(whole):
            fail_in.value = k
            assert status(lambda: t.set_attribute(14)) == {CUDA_ERROR}
            assert use() == {STATE}
            before = ctx.launches
            t.set_attribute(14)
            assert ctx.launches - before == whole and use() == 0
            t.set_attribute(0)
        print(whole)
        """, DCF_BASIN_MIN=least)
    assert int(said[0]) >= 4


@pytest.mark.parametrize("least", [1, 1 << 40])
def test_contexts_on_two_devices_of_one_process(run, least):
    """Opt-ins to more than 48 KB of shared memory hold for one device: a context on a
    second one needs its own, and so does one made after the device was reset."""
    said, rows = run("""
        def everything(device):
            ctx = dcf.Context(device)
            for attr in (0, 18, 14):
                t = ctx.build(np.zeros((300, 410), np.uint16), connectivity=8, tree_type="max", attribute=attr)
                t.filter(attr, 2.0)
                t.pattern_spectrum(attr, np.float32([0, 1, 2]))
            b = ctx.batch([(40, 50), (70, 33)], np.float32, connectivity=8, attribute=13)
            b.run(np.zeros(40 * 50 + 70 * 33, np.float32), filter_attr=0, lam=3.0, use_graph=False)
        everything(0)
        everything(1)
        C.CDLL(None).fake_reset()
        everything(1)
        """, DCF_BASIN_MIN=least)
    assert {r[0] for r in rows} == {0, 1}
    assert not [r for r in rows if r[2]]


@pytest.mark.parametrize("shape,conn", [((2_097_121, 1), 4), ((2_097_153, 2), 8), ((524_281, 1, 1), 6),
                                        ((524_289, 2, 1), 26), ((2, 1_048_561, 1), 6)])
def test_tall_images_are_built(run, shape, conn):
    """Rows and slices beyond 65535 tiles of them: no launch is refused."""
    said, rows = run(f"""
        ctx = dcf.Context(0)
        ctx.build(np.zeros({shape}, np.uint8), connectivity={conn}, tree_type="max", attribute=0)
        """)
    assert len(rows) > 15 and not [r for r in rows if r[2]]


def test_merging_build_refuses_what_its_launch_cannot_hold(run):
    """The merging build's tiles are a plain 3-D grid: taller images end at its tile kernel."""
    said, rows = run("""
        ctx = dcf.Context(0)
        print(status(lambda: ctx.build(np.zeros((2_097_121, 1), np.uint8), connectivity=4, tree_type="max", attribute=0)))
        """, DCF_BASIN_MIN=1 << 40)
    assert said == [str(CUDA_ERROR)] and [r[2] != 0 for r in rows] == [False] * (len(rows) - 1) + [True]
    assert "k_tile_build" in rows[-1][1]


@pytest.mark.parametrize("n", [1, 441, 3584, 3585, 4096, 4097])
@pytest.mark.parametrize("dtype", ["uint16", "float32"])
def test_spectra_have_room_beside_static_shared_memory(run, dtype, n):
    """k_spectrum<true> has its thresholds in static shared memory (6144 bytes): with the
    histogram that may be more than a kernel gets without an opt-in."""
    said, rows = run(f"""
        ctx = dcf.Context(0)
        t = ctx.build(np.zeros((50, 60), np.{dtype}), connectivity=8, tree_type="max", attribute=18)
        t.pattern_spectrum(18, np.arange({n}, dtype=np.float32))
        """)
    device, name, status, dynamic, opted = rows[-1]
    assert "k_spectrum" in name and status == 0
    assert opted or dynamic + 6144 <= 48 * 1024


def test_autotuner_leaves_what_it_cannot_measure(run):
    """Nothing of a basin batch's build depends on the schedule: the tuner times the build
    once and keeps the schedule, which governs the spectrum's tile walk.  A merging batch
    is tuned as ever."""
    code = """
        ctx = dcf.Context(0)
        b = ctx.batch([(300, 410), (70, 33)], np.float32, connectivity=8, attribute=13)
        pix = np.zeros(300 * 410 + 70 * 33, np.float32)
        b.set_schedule((128, 32), 1, 2)
        b.set_merge(seam_buckets=8, up_steps=77)
        before = b.info()
        ms = b.autotune(pix, repeats=2)
        after = b.info()
        print(ms, int(all(before[k] == after[k] for k in ("tile", "ctas_per_sm", "chunk", "seam_buckets", "up_steps"))))
        """
    said, rows = run(code)
    assert said == ["1.0", "1"]
    assert sum("k_basins" in r[1] for r in rows) == 3  # a warm-up and two repeats
    said, rows = run(code, DCF_BASIN_MIN=1 << 40)
    assert float(said[0]) == 1.0 and sum("k_batch_tile_build" in r[1] for r in rows) > 10


def test_min_rule_without_room_for_the_chains_scratch(run):
    """The min rule along the chains wants 8 bytes a pixel at once and a value a chain; with
    less free than that, but enough for what the general path still lacks after a max filter
    (4 + 4 bytes a pixel), it takes that one."""
    said, rows = run("""
        n = 400 * 500
        ctx = dcf.Context(0)
        t = ctx.build(np.zeros((400, 500), np.uint16), connectivity=4, tree_type="max", attribute=0)
        memory.value = in_use.value  # full: the next allocation takes the build's scratch back
        t.filter(0, 5.0, "max")
        memory.value = in_use.value + 8 * n + 4096
        print(status(lambda: t.filter(0, 5.0, "min")))
        """)
    assert said == ["0"]
    assert any("k_jump_last" in r[1] for r in rows)


BATCH = """
shapes = [(1000, 1400), (700, 900)]
n = sum(h * w for h, w in shapes)
pix = np.zeros(n, np.float32)
lv = np.float32([0, 1, 2])
ctx = dcf.Context(0)
b = ctx.batch(shapes, np.float32, connectivity=8, attribute=13)
ops = dict(filter_attr=0, lam=3.0, spectrum=(13, lv, 0, lv))
"""


def test_batch_gives_its_scratch_back_for_its_own_buffers(run):
    """Room for less than a run's buffers beside the basin scratch: the batch merges."""
    said, rows = run(BATCH + """
memory.value = in_use.value + n
for graph in (False, True, True):
    print(status(lambda: b.run(pix, use_graph=graph, **ops)))
    print(status(lambda: b.adjoint(np.ones(n, np.float32), np.ones((2, 3, 3)))))
print(status(lambda: b.autotune(pix, repeats=1)))
""")
    assert said == ["0"] * 7
    assert not any("k_basins" in r[1] for r in rows) and any("k_batch_tile_build" in r[1] for r in rows)


def test_batch_gives_its_scratch_back_after_a_run(run):
    """The gradient, the parents or a tree that finds no room takes an idle batch's scratch;
    another batch's own scratch does not."""
    for call in ("b.adjoint(np.ones(n, np.float32), np.ones((2, 3, 3)))", "b.parent()", "b.node_attribute(13)",
                 "ctx.build(np.zeros((1000, 800), np.float32), connectivity=8, tree_type='max', attribute=13)"):
        said, rows = run(BATCH + f"""
print(status(lambda: b.run(pix, use_graph=False, **ops)))
memory.value = in_use.value + n
print(status(lambda: {call}))
print(ctx.launches)
print(status(lambda: b.run(pix, use_graph=False, **ops)))
""")
        assert [said[i] for i in (0, 1, 3)] == ["0"] * 3, call
        later = "".join(r[1] for r in rows[int(said[2]):])
        assert "k_batch_tile_build" in later and "k_basins" not in later, call
    said, rows = run(BATCH + """
memory.value = in_use.value + 120 * n  # room for another batch without the scratch
c = ctx.batch(shapes, np.float32, connectivity=8, attribute=13)
at = ctx.launches
print(status(lambda: c.run(pix, use_graph=False)), status(lambda: b.run(pix, use_graph=False)))
""")
    names = [r[1] for r in rows]
    assert said == ["0", "0"]
    assert sum("k_batch_tile_build" in k for k in names) == 1 and sum("k_basins" in k for k in names) == 1
