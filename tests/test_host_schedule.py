"""Which kernels the C ABI runs on which states, checked without a GPU: the
library's host objects on a device of host memory (drivers/host_device.cu),
whose levels know when a kernel reads a state that it must not."""
import ctypes as C
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import numpy as np
import pytest

import lbm3_b200 as L
from lbm3_b200 import _abi as A
from lbm3_b200 import build as B

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    B.build()
    out = tmp_path_factory.mktemp("host") / "host_device.so"
    objs = [str(B.OBJ_DIR / o) for o in ("api.o", "builder.o", "geometry.o")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I/usr/local/cuda/include",
                    "-Wl,-Bsymbolic", str(ROOT / "tests" / "drivers" / "host_device.cpp"), *objs, "-o", str(out)],
                   check=True)
    lib = C.CDLL(str(out))
    for name, res, args in A.SIGNATURES:
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    for name in ("cudaStreamBeginCapture", "cudaGraphLaunch", "cudaGraphInstantiate", "cudaStreamEndCapture"):
        getattr(lib, name).restype = C.c_int
    lib.host_device_pitch_limit.argtypes = [C.c_size_t]
    return lib


@pytest.fixture
def device(library, monkeypatch):
    """device(ghosts): an empty device whose new levels' ghosts repeat their sources, or do not."""
    monkeypatch.setattr(A, "lib", lambda: library)

    def reset(ghosts):
        library.host_device_reset(int(ghosts))
        return library
    return reset


def level(lib, order=0):
    """{steps, ghosts repeat their sources, ghost exchange due, read in a wrong state}"""
    out = (C.c_int * 4)()
    assert lib.host_device_level(order, out) == 0
    return dict(zip(("steps", "ghosts", "due", "wrong"), out))


def done(steps):
    """An ordinary state after `steps` steps, on which every kernel may run."""
    return {"steps": steps, "ghosts": 1, "due": 0, "wrong": 0}


class Captured:
    """Work on `stream` inside the block is recorded; replay() runs it."""

    def __init__(self, lib, stream):
        self.lib, self.stream, self.exec = lib, C.c_void_p(stream), C.c_void_p()

    def __enter__(self):
        assert self.lib.cudaStreamBeginCapture(self.stream, 0) == 0
        return self

    def __exit__(self, *exc):
        graph = C.c_void_p()
        assert self.lib.cudaStreamEndCapture(self.stream, C.byref(graph)) == 0
        assert self.lib.cudaGraphInstantiate(C.byref(self.exec), graph, C.c_ulonglong(0)) == 0

    def replay(self):
        assert self.lib.cudaGraphLaunch(self.exec, self.stream) == 0


@pytest.mark.parametrize("ghosts", [False, True])
@pytest.mark.parametrize("call", ["single", "pairs", "update_batch", "packed"])
def test_captured_steps_replay_on_any_state(device, call, ghosts):
    """A program's own graph of steps does not know the state that it is
    replayed on: after new populations, their ghosts differ from their sources."""
    lib = device(ghosts)
    with L.build_grids(L.periodic_box(6, 4, 4)) as g:
        g.set_stream(64)
        batch = L.PackedBatch([g]) if call == "packed" else None
        with Captured(lib, 64) as c:
            if call == "single":
                g.update_all_grids(1)
                g.update_all_grids(1)
            elif call == "pairs":
                g.update_all_grids(2)
            elif call == "update_batch":
                L.update_batch([g], 2)
            else:
                batch.update(2)
        assert level(lib)["steps"] == 0
        for n in (1, 2):
            g.set_populations(g.populations())
            c.replay()
            assert level(lib) == done(2 * n)
        # and steps outside of it go on from there
        g.update_all_grids(3)
        assert level(lib) == done(7)
        if batch:
            batch.close()


@pytest.mark.parametrize("ghosts", [False, True])
@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5])
def test_states_between_calls(device, steps, ghosts):
    """Every division of steps over the entry points leaves an ordinary state."""
    lib = device(ghosts)
    grids = [L.build_grids(L.periodic_box(6, 4, 4 + 2 * q)) for q in range(3)]
    with L.PackedBatch(grids[1:]) as b:
        for k in range(2):
            grids[0].update_all_grids(steps)
            b.update(steps)
            L.update_batch(grids, steps)
            for g in grids:
                g.macro()
                g.kinetic_energy(1.0, 1.0)
            assert [level(lib, q) for q in range(3)] == [done(2 * (k + 1) * steps)] * 3
    for g in grids:
        g.close()


@pytest.mark.parametrize("call", ["update", "time_steps"])
def test_no_steps_change_nothing(device, call):
    """A batch advanced by no steps: ghosts that differ from their sources
    still differ, and the next step copies them."""
    lib = device(False)
    with L.build_grids(L.periodic_box(6, 4, 4)) as g, L.build_grids(L.open_channel(8, 6, 6)) as other:
        with L.PackedBatch([g, other]) as b:
            getattr(b, call)(0)
            assert (level(lib)["steps"], level(lib)["ghosts"]) == (0, 0)
            b.update(2)
        assert level(lib) == done(2)


def test_two_threads_read_one_object(device):
    """Fields and populations of the levels of one object, read by two host
    threads at once, each come out as from one thread."""
    lib = device(True)
    with L.build_grids(L.taylor_green_refined(16).case) as g:
        reads = [lambda: g.macro(0), lambda: g.populations(1), lambda: g.macro(1)]
        alone = [r() for r in reads]
        lib.host_device_copy_delay(2000)  # between a read's kernel and its copy
        with ThreadPoolExecutor(3) as pool:
            for _ in range(3):
                for a, b in zip(alone, pool.map(lambda r: r(), reads)):
                    np.testing.assert_array_equal(a, b)


def test_fields_wider_than_a_pitched_copy(device):
    """Fields of several staging pieces whose row is longer than the pitch that
    a 2D copy may have (2^31 - 1 bytes; here 1 MiB, for a level that fits a test)."""
    device(True).host_device_pitch_limit(1 << 20)
    with L.build_grids(L.periodic_box(64, 64, 64)) as g:
        m = g.macro()
        assert m[0].nbytes > 1 << 20
        cells = np.arange(m.shape[1], dtype=np.float32) * 16
        np.testing.assert_array_equal(m, cells + 4 * np.arange(4, dtype=np.float32)[:, None])


@pytest.mark.parametrize("ghosts", [False, True])
@pytest.mark.parametrize("graphs", [0, 1, 2])
@pytest.mark.parametrize("call", ["single", "update_batch", "packed"])
def test_a_failed_call_leaves_ordinary_states(device, call, graphs, ghosts):
    """The runtime refuses a graph in the middle of a call: the steps that ran
    are counted, and every domain is left in a state that readers may use."""
    lib = device(ghosts)
    # the last one steps without graphs, and is therefore stepped in any case
    grids = [L.build_grids(L.periodic_box(6, 4, 4 + 2 * q)) for q in range(3)]
    grids[2].set_graphs(call == "packed")
    batch = L.PackedBatch(grids) if call == "packed" else None
    lib.host_device_instantiations(graphs)

    def advance(n):
        try:
            if batch:
                batch.update(n)
            elif call == "update_batch":
                L.update_batch([grids[2], *grids[:2]], n)
            else:
                for g in grids:
                    g.update_all_grids(n)
        except A.LbmError:
            return False
        return True

    enough = {"single": 2, "update_batch": 2, "packed": 1}[call]
    assert advance(7) == (graphs >= enough)
    for q, g in enumerate(grids):
        assert level(lib, q) == {**done(g.info().iterations_finished), "ghosts": level(lib, q)["ghosts"]}
        g.macro()
    lib.host_device_instantiations(-1)
    before = [g.info().iterations_finished for g in grids]
    if batch:
        assert len(set(before)) == 1
    assert advance(5)
    for q, g in enumerate(grids):
        assert level(lib, q) == done(before[q] + 5)
    if batch:
        batch.close()
    for g in grids:
        g.close()


def test_a_failed_write_leaves_ghosts_unknown(device):
    """Populations written in part: the next step copies the ghosts."""
    lib = device(True)
    with L.build_grids(L.periodic_box(64, 64, 64)) as g:
        f = g.populations()
        lib.host_device_uploads(3)
        with pytest.raises(A.LbmError):
            g.set_populations(f)
        lib.host_device_uploads(-1)
        g.update_all_grids(2)
        assert level(lib) == done(2)


@pytest.mark.parametrize("stale", [0, 1, 20])
def test_launches_of_a_one_step_batch_call(device, stale):
    """A packed batch of 20 periodic boxes, one step per call: two launches for
    the step (16 domains each) and two for the ghost exchange; two (collision
    and ghost copies) for the members with new populations, however many."""
    lib = device(True)
    grids = [L.build_grids(L.periodic_box(4, 4, 4)) for _ in range(20)]
    with L.PackedBatch(grids) as b:
        for n, changed in enumerate((0, stale, 0)):
            for g in grids[:changed]:
                g.set_populations(g.populations())
            before = lib.host_device_launches()
            b.update(1)
            fresh = 20 - changed
            assert lib.host_device_launches() - before == 2 * -(-fresh // 16) + (2 if changed else 0)
            assert [level(lib, q) for q in range(20)] == [done(n + 1)] * 20
    for g in grids:
        g.close()
