"""The solver's host side over a fake CUDA runtime (fake_cuda.cpp): failing
allocations and the routes that calls take, on the CPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

import fim_api
import fim_mesh

STAGE, ARENA, NBR, EVEC = range(4)
OOM = 7


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    src = os.path.join(PKG, "csrc", "fim_solver.cpp")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wall", "-Wno-subobject-linkage", "-I" + os.path.join(cuda, "include"),
                           f'-DFIM_SOLVER_CPP="{src}"', os.path.join(ROOT, "tests", "fake_cuda.cpp"), "-o", out,
                           "-Wl,--no-undefined,-Bsymbolic"])  # (its own runtime, not one that torch has loaded)
    lib = C.CDLL(out)
    vp, i64, sz = C.c_void_p, C.c_int64, C.c_size_t
    lib.fim_create.argtypes = [vp, C.POINTER(vp)]
    lib.fim_destroy.argtypes = [vp]
    lib.fim_last_error.argtypes = [vp]
    lib.fim_last_error.restype = C.c_char_p
    for f in (lib.fim_set_mesh, lib.fim_set_mesh_i32):
        f.argtypes = [vp, i64, vp, i64, vp, vp]
    lib.fim_set_conduction.argtypes = lib.fim_set_conduction_device.argtypes = [vp, vp, vp, vp]
    lib.fim_set_stimuli.argtypes = [vp, i64, vp, vp]
    lib.fim_solve.argtypes = [vp, vp]
    lib.fim_get_times.argtypes = [vp, vp, vp]
    lib.fake_budget.argtypes = [sz]
    lib.fake_live.restype = lib.fake_peak.restype = lib.fake_bytes.restype = sz
    lib.fake_bytes.argtypes = [vp, C.c_int]
    lib.fake_lists.argtypes = [vp, C.POINTER(C.c_ulonglong)]
    lib.fake_front_width.argtypes = [vp]
    lib.fake_front_width.restype = C.c_double
    lib.fake_metric_reads.argtypes = [vp]
    return lib


def ptr(a):
    return None if a is None else C.c_void_p(a.ctypes.data)


class Solver:
    def __init__(self, L):
        self.L, self.h = L, C.c_void_p()
        L.fake_budget(2 ** 62)
        assert L.fim_create(None, C.byref(self.h)) == 0
        self.idle = L.fake_live()

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.L.fim_destroy(self.h)
        assert self.L.fake_live() == 0
        self.L.fake_budget(2 ** 62)

    def room(self, n):
        """n bytes beyond what the solver holds without a mesh."""
        self.L.fake_budget(self.idle + n)

    def set_mesh(self, m):
        xyz, tets, tags = m
        f = self.L.fim_set_mesh_i32 if tets.dtype == np.int32 else self.L.fim_set_mesh
        return f(self.h, len(xyz), ptr(xyz), len(tets), ptr(tets), ptr(tags))

    def bytes(self, k):
        return self.L.fake_bytes(self.h, k)

    def lists(self):
        out = C.c_ulonglong()
        self.L.fake_lists(self.h, C.byref(out))
        return out.value, self.L.fake_front_width(self.h)

    def solve(self, nV, nT):
        one = np.ones(3 * nT)
        v, t = np.zeros(1, dtype=np.int64), np.zeros(1)
        for rc in (self.L.fim_set_conduction(self.h, ptr(one), ptr(one), ptr(one)),
                   self.L.fim_set_stimuli(self.h, 1, ptr(v), ptr(t)), self.L.fim_solve(self.h, None)):
            assert rc == 0, self.L.fim_last_error(self.h)

    def times(self, nV):
        phi, st = np.full(nV, -1.0), np.full(nV, -1, dtype=np.int32)
        rc = self.L.fim_get_times(self.h, ptr(phi), ptr(st))
        assert rc == 0, self.L.fim_last_error(self.h)
        assert np.array_equal(phi, 0.5 * np.arange(nV)) and np.array_equal(st, np.arange(nV) % 6)


def mesh(cells, ids=np.int64, tagged=False, seed=1):
    xyz, tets = fim_mesh.kuhn_box(*cells, *[0.1 * c for c in cells], seed=seed)
    tags = (np.arange(len(tets)) * 3 // len(tets)).astype(np.int32) if tagged else None
    return np.ascontiguousarray(xyz, dtype=np.float64), np.ascontiguousarray(tets, dtype=ids), tags


def test_a_failed_allocation_is_reported_once(L):
    """Where a mesh finds no room to be staged, the one in place still solves
    and reads back, above the size from which reading back launches a kernel;
    a mesh that does fit is then accepted."""
    m, big, small = mesh((33, 25, 19)), mesh((60, 40, 30)), mesh((4, 3, 2))
    nV, nT = len(m[0]), len(m[1])
    assert nV > 16384
    with Solver(L) as s:
        assert s.set_mesh(m) == 0
        s.solve(nV, nT)
        L.fake_budget(L.fake_live() + 4096)  # (no room for the big one's staging)
        bad = (big[0], np.where(big[1] == 7, len(big[0]), big[1]), None)
        assert s.set_mesh(bad) != 0
        s.times(nV)
        s.solve(nV, nT)
        s.times(nV)
        assert s.set_mesh(small) == 0, L.fim_last_error(s.h)


@pytest.mark.parametrize("tagged", [False, True])
@pytest.mark.parametrize("short", ["evec", "nbr"])
def test_edge_vectors_give_way(L, tagged, short):
    """The edge vectors are optional: a mesh for which they leave no room, or
    which leaves none for them, is staged without them, with the same lists."""
    m = mesh((7, 5, 4), tagged=tagged)
    with Solver(L) as s:
        assert s.set_mesh(m) == 0
        want, need = s.lists(), [s.bytes(k) for k in range(4)]
    assert need[EVEC] == 144 * len(m[1])
    with Solver(L) as s:
        # all but one byte of what everything takes, and all but the edge vectors
        s.room(sum(need) - 1 if short == "evec" else sum(need) - need[EVEC])
        assert s.set_mesh(m) == 0, L.fim_last_error(s.h)
        assert s.bytes(EVEC) in (0, need[EVEC]) and s.lists() == want


@pytest.mark.parametrize("ids", [np.int64, np.int32])
@pytest.mark.parametrize("tagged", [False, True])
@pytest.mark.parametrize("cells", [(1, 1, 1), (7, 5, 4)])
def test_staging_takes_no_room_from_the_mesh(L, cells, tagged, ids):
    """A mesh fits where its own arrays fit, with or without one in place, and
    the edge vectors where these fit too: the staging buffer is given up for
    either, and the lists are the same."""
    m, other = mesh(cells, ids, tagged), mesh(cells, ids, tagged, seed=2)
    with Solver(L) as s:
        assert s.set_mesh(other) == 0
        want_other = s.lists()
        assert s.set_mesh(m) == 0
        want, need = s.lists(), [s.bytes(k) for k in range(4)]
    mine = need[ARENA] + need[NBR]
    far = (np.concatenate([m[0], np.ones((50, 3))]), m[1], m[2])  # more vertices than copies
    with Solver(L) as s:
        assert s.set_mesh(far) == 0
        want_far, far_mine = s.lists(), s.bytes(ARENA) + s.bytes(NBR)
    for room, evec in ((mine, 0), (mine + need[EVEC], need[EVEC])):
        with Solver(L) as s:
            s.room(room)
            for k in range(2):
                assert s.set_mesh(m) == 0, L.fim_last_error(s.h)
                assert s.lists() == want and s.bytes(EVEC) == evec and s.bytes(STAGE) == 0
                # a rejected mesh leaves this one, without room to check it on the device too
                bad = m[1].copy()
                bad[-1, 2] = bad[-1, 1]
                assert s.set_mesh((m[0], bad, m[2])) == 1
                assert f"tet {len(bad) - 1} repeats".encode() in L.fim_last_error(s.h)
                bad[0, 3] = len(m[0])
                assert s.set_mesh((m[0], bad, m[2])) == 1 and b"tet 0 has vertex" in L.fim_last_error(s.h)
                nan = m[0].copy()
                nan[1, 1] = np.nan
                assert s.set_mesh((nan, m[1], m[2])) == 1 and b"coordinate 4 " in L.fim_last_error(s.h)
                assert s.lists() == want
                s.room(room)
                assert s.set_mesh(other) == 0 and s.lists() == want_other
    with Solver(L) as s:
        s.room(far_mine)
        assert s.set_mesh(far) == 0, L.fim_last_error(s.h)
        assert s.lists() == want_far
    with Solver(L) as s:
        s.room(far_mine - 1)
        assert s.set_mesh(far) == OOM and b"out of memory" in L.fim_last_error(s.h)


def test_a_larger_mesh_replaces_a_smaller_one(L):
    """What is left of the previous mesh makes room for the next one's arrays."""
    a, b = mesh((7, 5, 4)), mesh((11, 8, 6))
    with Solver(L) as s:
        assert s.set_mesh(b) == 0
        want, need = s.lists(), [s.bytes(k) for k in range(4)]
    with Solver(L) as s:
        s.room(need[ARENA] + need[NBR])
        assert s.set_mesh(a) == 0 and s.bytes(EVEC) > 0 and s.bytes(STAGE) > 0
        assert s.set_mesh(b) == 0, L.fim_last_error(s.h)
        assert s.lists() == want


@pytest.mark.parametrize("device,in_place", [(0, True), (1, False)])
def test_a_field_on_another_device_is_copied(L, device, in_place):
    """The metric kernel reads a field where it is only on the solver's own
    device; from another one it goes through the copies."""
    m = mesh((4, 3, 2))
    with Solver(L) as s:
        assert s.set_mesh(m) == 0
        fib, cf = np.ones(3 * len(m[1])), np.ones(len(m[1]))
        L.fake_other_device(device)
        rc = L.fim_set_conduction_device(s.h, ptr(fib), ptr(cf), ptr(cf))
        L.fake_other_device(0)
        assert rc == 0 and bool(L.fake_metric_reads(ptr(fib))) == in_place


@pytest.mark.parametrize("nV", [16384, 16385, 60000, 140000])
@pytest.mark.parametrize("cells", [(1, 1, 1), (12, 10, 8), (30, 20, 12), (40, 30, 25)])
def test_states_of_a_few_tagged_tets_among_many_vertices(L, cells, nV):
    """States are read back in a few copies, however short the vertex lists
    are that the states are widened through."""
    xyz, tets, tags = mesh(cells, tagged=True)
    nV = max(nV, len(xyz))
    m = (np.concatenate([xyz, np.ones((nV - len(xyz), 3))]), tets, tags)
    with Solver(L) as s:
        assert s.set_mesh(m) == 0
        s.solve(nV, len(tets))
        L.fake_d2h()
        s.times(nV)
        assert L.fake_d2h() <= 5
