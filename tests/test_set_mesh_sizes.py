"""A mesh that the library rejects leaves the previous one in place, and the
binding's sizes (which times() allocates by) with it."""
from types import SimpleNamespace

import numpy as np
import pytest

import fim_api


@pytest.mark.parametrize("ids", [np.int32, np.int64])
@pytest.mark.parametrize("n", [4, 400])
def test_rejected_mesh_keeps_the_sizes(monkeypatch, ids, n):
    s = object.__new__(fim_api.Solver)
    s.h, s.nV, s.nT = None, 40, 7
    monkeypatch.setattr(fim_api, "lib", lambda: SimpleNamespace(
        fim_set_mesh=lambda *a: 1, fim_set_mesh_i32=lambda *a: 1, fim_last_error=lambda h: b"rejected"))
    with pytest.raises(fim_api.FimError):
        s.set_mesh(np.zeros((n, 3)), np.zeros((n, 4), dtype=ids))
    assert (s.nV, s.nT) == (40, 7)


def test_accepted_mesh_sets_the_sizes(monkeypatch):
    s = object.__new__(fim_api.Solver)
    s.h, s.nV, s.nT = None, 0, 0
    monkeypatch.setattr(fim_api, "lib", lambda: SimpleNamespace(fim_set_mesh=lambda *a: 0))
    s.set_mesh(np.zeros((9, 3)), np.zeros((5, 4), dtype=np.int64))
    assert (s.nV, s.nT) == (9, 5)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 5000])
def test_times_after_a_rejected_mesh(built_library, n):
    """Fewer and more vertices than the mesh in place: it solves and reads back as before."""
    import fim_mesh
    c = fim_mesh.cube_case(5)
    rng = np.random.default_rng(n)
    with fim_api.Solver() as s:
        s.set_mesh(c["xyz"], c["tets"])
        s.set_conduction(c["fib"], c["cf"], c["ct"])
        s.set_stimuli(c["seed_v"], c["seed_t"])
        s.solve()
        phi, st = s.times()
        with pytest.raises(fim_api.FimError):
            s.set_mesh(rng.normal(size=(n, 3)), np.array([[0, 1, 2, n]]))
        got = s.times()
        assert np.array_equal(got[0], phi) and np.array_equal(got[1], st)
        s.solve()
        got = s.times()
        assert np.array_equal(got[0], phi) and np.array_equal(got[1], st)
