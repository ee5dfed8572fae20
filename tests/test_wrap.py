"""The ghost-free periodic step's rule, checked on the host: reading across a
periodic face from the cell's own image, with one ghost exchange at the end,
leaves exactly the state that ghost copies after every step leave; and only
levels on which that holds qualify."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

import lbm3_b200 as L
from lbm3_b200 import build as B
from lbm3_b200 import geometry as G

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    B.build()
    out = tmp_path_factory.mktemp("wrap") / "wrap_check.so"
    objs = [str(B.OBJ_DIR / "builder.o"), str(B.OBJ_DIR / "geometry.o")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "drivers" / "wrap_check.cpp"), *objs, "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.lbm_wrap_check.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_longlong)]

    def run(case, steps):
        skipped = C.c_longlong()
        return lib.lbm_wrap_check(C.byref(case), steps, C.byref(skipped)), skipped.value
    return run


def _rotor(n, origin=(0.0, 0.0, 0.0)):
    c = L.periodic_box(n, n, n - 4)
    tris = G.rotor(hub_radius=2, tip_radius=6, chord=3, thickness=1.0, hub_length=4, center=origin)
    return G.set_rotors(c, [(tris, dict(axis=2, origin=origin, radians_per_second=2.0))])


@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 2, 6), (6, 10, 4), (16, 8, 12), (34, 6, 2)])
@pytest.mark.parametrize("steps", [1, 2, 5])
def test_same_state_as_ghost_copies(check, dims, steps):
    assert check(L.periodic_box(*dims), steps) == (0, 0)


def test_rotor_cells_stay_out_of_the_tiles(check):
    status, skipped = check(_rotor(24), 3)
    assert status == 0 and skipped > 0


def _rejected():
    yield "rotor at a face", _rotor(24, (7.0, 0.0, 0.0))
    yield "open faces", L.open_channel(16, 8, 8, sides="periodic")
    walls = L.periodic_box(16, 16, 16)
    G.set_bodies(walls, [G.icosphere(2, 4.0, (0.0, 0.0, 0.0))])
    yield "walls", walls
    yield "refined", L.taylor_green_refined(16).case


@pytest.mark.parametrize("name,case", list(_rejected()))
def test_other_levels_do_not_qualify(check, name, case):
    assert check(case, 1)[0] == 2
