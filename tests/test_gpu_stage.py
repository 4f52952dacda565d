"""Mesh staging on the device (fim_set_mesh): the solve of the staged mesh
equals the oracle bit for bit at the sizes where the corner and neighbour
lists can go wrong -- a single tet, vertices in no tet, shuffled ids, and
hubs with more corners than one warp, the sorting buffer and the sorted runs
hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F(built_library):
    import fim_api
    return fim_api


@pytest.fixture(scope="module")
def O(oracle_lib):
    return oracle_lib


def fan(rings, sectors, seed=0, extra=0):
    """A ball of tets around one hub vertex: 2 * sectors * rings of them."""
    th = np.linspace(0.0, np.pi, rings + 2)[1:-1]
    ph = np.arange(sectors) * (2 * np.pi / sectors)
    ring = np.stack([np.outer(np.sin(th), np.cos(ph)), np.outer(np.sin(th), np.sin(ph)),
                     np.outer(np.cos(th), np.ones(sectors))], axis=-1).reshape(-1, 3)
    xyz = np.concatenate([[[0, 0, 0], [0, 0, 1.0], [0, 0, -1.0]], ring])
    tets = []
    for s in range(sectors):
        n = (s + 1) % sectors
        tets.append([0, 1, 3 + s, 3 + n])
        for r in range(rings - 1):
            a, b = 3 + r * sectors + s, 3 + r * sectors + n
            tets += [[0, a, b, a + sectors], [0, b, b + sectors, a + sectors]]
        last = 3 + (rings - 1) * sectors
        tets.append([0, 2, last + s, last + n])
    xyz = np.concatenate([xyz, np.full((extra, 3), 2.0)])  # vertices in no tet
    rng = np.random.default_rng(seed)
    perm = rng.permutation(len(xyz))
    out = np.empty_like(xyz)
    out[perm] = xyz
    tets = perm[np.array(tets)][rng.permutation(len(tets))]
    return out, rng.permuted(tets, axis=1).astype(np.int64)


def case_of(xyz, tets, seed=1):
    rng = np.random.default_rng(seed)
    nT = len(tets)
    f = rng.normal(size=(nT, 3))
    f /= np.linalg.norm(f, axis=1)[:, None]
    cf = rng.uniform(0.4, 0.8, size=nT)
    used = np.unique(tets)
    return dict(xyz=xyz, tets=tets, fib=f, cf=cf, ct=cf * rng.uniform(0.3, 0.6, size=nT),
                seed_v=rng.choice(used, size=2, replace=False), seed_t=np.array([0.0, 0.7]))


def check(F, O, s, c):
    s.set_mesh(c["xyz"], c["tets"])
    s.set_conduction(c["fib"], c["cf"], c["ct"])
    s.set_stimuli(c["seed_v"], c["seed_t"])
    s.solve()
    phi, st = s.times()
    nV = len(c["xyz"])
    slots, _, _, _ = O.reference_slots(nV, c["tets"], None)
    geo = O.metric_geo(slots, c["xyz"], c["fib"], c["cf"], c["ct"])
    phi_o, st_o, it_o, upd_o = O.solve_pure(nV, slots, geo, c["seed_v"], c["seed_t"])
    assert np.array_equal(phi, phi_o) and np.array_equal(st, st_o)
    stats = s.stats()
    assert stats["iterations"] == it_o and stats["vertex_updates"] == upd_o


@pytest.mark.parametrize("rings,sectors,extra", [(1, 3, 0), (2, 8, 5), (4, 10, 0), (9, 19, 0), (10, 18, 3),
                                                 (30, 40, 0)],
                         ids=["6", "32", "80", "342", "360", "2400"])
def test_hub_of_many_tets(F, O, rings, sectors, extra):
    xyz, tets = fan(rings, sectors, seed=rings, extra=extra)
    with F.Solver() as s:
        check(F, O, s, case_of(xyz, tets))


def test_single_tet_and_meshes_of_changing_size(F, O):
    """One solver over meshes that grow and shrink (kept buffers)."""
    import fim_mesh
    one = (np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]]), np.array([[2, 0, 3, 1]]))
    big = fim_mesh.kuhn_box(17, 9, 7, 1.7, 0.9, 0.7, seed=4)
    with F.Solver() as s:
        for xyz, tets in (one, fan(5, 12), big, one, fan(3, 7, extra=40), big):
            check(F, O, s, case_of(xyz, np.asarray(tets, dtype=np.int64)))


def test_rejected_mesh_leaves_the_previous_one(F, O):
    xyz, tets = fan(4, 9)
    c = case_of(xyz, tets)
    with F.Solver() as s:
        check(F, O, s, c)
        phi = s.times(with_state=False)
        out, twice, nan = tets.copy(), tets.copy(), xyz.copy()
        out[7, 2] = len(xyz)
        out[9, 0] = -1
        twice[3, 1] = twice[3, 0]
        nan[5, 1] = np.nan
        both = out.copy()
        both[2, 3] = both[2, 0]
        for bad_xyz, bad_tets, text in ((xyz, out, f"tet 7 has vertex {len(xyz)}"), (xyz, twice, "tet 3 repeats"),
                                        (nan, tets, "coordinate 16 "), (nan, both, "tet 7 has vertex"),
                                        (nan, twice, "tet 3 repeats")):
            with pytest.raises(F.FimError, match=text):
                s.set_mesh(bad_xyz, bad_tets)
        s.nV, s.nT = len(xyz), len(tets)
        s.solve()
        assert np.array_equal(s.times(with_state=False), phi)


@pytest.mark.parametrize("tagged", [False, True])
def test_ids_of_32_and_64_bits(F, O, tagged):
    """Meshes with ids of either width, in any layout, solve to the same bits;
    a bad id is reported the same way."""
    import fim_mesh
    xyz, tets = fim_mesh.kuhn_box(9, 5, 4, 1.0, 0.6, 0.5, seed=2)
    c = case_of(xyz, np.asarray(tets, dtype=np.int64))
    tags = (np.arange(len(tets)) * 3 // len(tets)).astype(np.int32) if tagged else None
    wide = np.asarray(tets, dtype=np.int64)
    strided = np.zeros((len(tets), 8), dtype=np.int32)
    strided[:, ::2] = wide
    got = []
    for ids in (wide, wide.astype(np.int32), strided[:, ::2], np.asfortranarray(wide.astype(np.int32)),
                wide.astype(np.uint32), wide.astype(np.int16)):
        with F.Solver() as s:
            s.set_mesh(xyz, ids, tags)
            s.set_conduction(c["fib"], c["cf"], c["ct"])
            s.set_stimuli(c["seed_v"], c["seed_t"])
            s.solve()
            got.append(s.times())
            bad = np.array(ids)
            bad[5, 3] = len(xyz)
            with pytest.raises(F.FimError, match=f"tet 5 has vertex {len(xyz)}"):
                s.set_mesh(xyz, bad, tags)
    for phi, st in got[1:]:
        assert np.array_equal(phi, got[0][0]) and np.array_equal(st, got[0][1])


@pytest.mark.parametrize("extra", [0, 3, 16384, 16387, 40000])  # states are widened on the device above 16,384 vertices
def test_states_of_vertices_in_no_tet(F, extra):
    """States come back for every vertex: with tags and more vertices in no
    tet than vertex copies too (they stay far, and unreached)."""
    import fim_mesh
    xyz, tets = fim_mesh.kuhn_box(5, 4, 3, 1.0, 0.8, 0.6, seed=3)
    n = len(xyz)
    c = case_of(xyz, np.asarray(tets, dtype=np.int64))
    tags = (np.arange(len(tets)) * 2 // len(tets)).astype(np.int32)
    far = np.concatenate([xyz, np.full((extra, 3), 9.0)])
    for at in (None, tags):
        got = []
        for points in (xyz, far):
            with F.Solver() as s:
                s.set_mesh(points, c["tets"], at)
                s.set_conduction(c["fib"], c["cf"], c["ct"])
                s.set_stimuli(c["seed_v"], c["seed_t"])
                s.solve()
                got.append(s.times())
        assert np.array_equal(got[1][0][:n], got[0][0]) and np.array_equal(got[1][1][:n], got[0][1])
        assert (got[1][1][n:] == F.FAR).all() and (got[1][0][n:] > 1e300).all()
        assert len(np.unique(got[0][1])) >= 1 and got[0][1].min() >= 0


@pytest.mark.parametrize("extra", [0, 3, 16387])
def test_states_are_the_oracles(F, O, extra):
    """States of a mesh with vertices in no tet, read back as bytes and widened
    on the device: the oracle's, far for those."""
    import fim_mesh
    xyz, tets = fim_mesh.kuhn_box(5, 4, 3, 1.0, 0.8, 0.6, seed=3)
    c = case_of(np.concatenate([xyz, np.full((extra, 3), 9.0)]), np.asarray(tets, dtype=np.int64))
    with F.Solver() as s:
        check(F, O, s, c)
        st = s.times()[1]
    assert set(np.unique(st[:len(xyz)])) == {F.FROZEN} and (st[len(xyz):] == F.FAR).all()
