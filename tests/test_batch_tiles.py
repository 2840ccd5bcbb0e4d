"""A batch's element tiles: the instance each tile's launch indexes the control blocks
and the time-step factors with.  Instances are padded to 128 elements; with
smaller blocks the last tiles of an instance may hold padding alone."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, assert_bitwise

SIDES = (1, 2, 5, 7, 9, 13, 20, 25)  # 20^3 = 62.5 and 25^3 = 122.07 default blocks

SHIM = r'''
#include "sgh_device.h"
extern "C" int code(int instance, int padding) { return padding ? fierro::padding_code(instance) : instance; }
extern "C" int tile(const int* inst, int t, int block) { return fierro::tile_instance(inst, t, block); }
'''


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    (d / "shim.cpp").write_text(SHIM)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", cuda, "-I",
                    os.path.join(ROOT, "fierro_gb300", "csrc"), str(d / "shim.cpp"), "-o", str(d / "libtiles.so")],
                   check=True)
    lib = C.CDLL(str(d / "libtiles.so"))
    lib.tile.argtypes = [C.c_void_p, C.c_int, C.c_int]
    return lib


@pytest.mark.parametrize("block", [32, 64, 128])
def test_every_tile_indexes_its_own_instance(tiles, block):
    ne = [n ** 3 for n in SIDES]
    inst, owner = [], []
    for i, n in enumerate(ne):
        pad = -n % 128
        inst += [tiles.code(i, 0)] * n + [tiles.code(i, 1)] * pad
        owner += [i] * ((n + pad) // block)
    inst = np.array(inst, dtype=np.int32)
    got = [tiles.tile(inst.ctypes.data, t, block) for t in range(inst.size // block)]
    assert got == owner
    assert block == 128 or (inst[::block] < 0).any()  # the case is met
    assert (inst < 0).sum() == sum(-n % 128 for n in ne)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("block", [None, 32, 64, 128])
def test_members_with_tiles_of_padding(lib_built, mode, block):
    from fierro_gb300 import problems, sgh
    ps = [problems.noh(n, jitter=0.05, seed=n, permute=True, cycles=10) for n in (1, 7, 13, 7)]
    ps[1].params.time_final = 0.004  # stops early
    states = [sgh.setup(p) for p in ps]
    with sgh.Batch(ps, fp_mode=mode) as b:
        if block:
            b.set_shape(128, 256, block, 0)
        for i, st in enumerate(states):
            b.set_state(i, st)
        b.run(10)
        got = [(sgh.compared_fields(b.get_state(i)), b.time(i)) for i in range(len(b))]
    for i, p in enumerate(ps):
        with sgh.SGHSolver(p, fp_mode=mode) as s:
            s.set_state(states[i])
            s.run(10)
            t = s.time()
            assert got[i][1] == (t[0], t[1], t[3])
            assert_bitwise(got[i][0], sgh.compared_fields(s.get_state()), list(got[i][0]), label="member %d" % i)
