"""The metric kernel's shorter forms (fibres in the xy-plane, along an axis)
and its general one: solves equal the oracle, whose norms are evaluated in
full, bit for bit -- also where forms meet inside a warp, with edges of no
length, and for fields the kernel reads in place or through a copy."""
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


def fibres(kind, n, rng):
    a = rng.uniform(-np.pi, np.pi, size=n)
    plane = np.stack([np.cos(a), np.sin(a), np.zeros(n)], axis=1)
    axis = np.zeros((n, 3))
    axis[np.arange(n), rng.integers(0, 2, size=n)] = rng.choice([-1.0, 1.0], size=n)
    full = rng.normal(size=(n, 3))
    full /= np.linalg.norm(full, axis=1)[:, None]
    if kind == "mixed":
        pick = rng.integers(0, 40, size=n)  # most warps hold more than one form
        return np.where((pick < 20)[:, None], plane, np.where((pick < 38)[:, None], axis, full))
    f = {"plane": plane, "axis": axis, "full": full}[kind]
    if kind == "plane":
        f[::7, 2] = -0.0
    return f


@pytest.mark.parametrize("kind", ["plane", "axis", "full", "mixed"])
@pytest.mark.parametrize("squash", [False, True])
def test_every_form_equals_the_oracle(F, O, kind, squash):
    import fim_mesh
    rng = np.random.default_rng(len(kind) + 10 * squash)
    xyz, tets = fim_mesh.kuhn_box(13, 7, 5, 1.3, 0.7, 0.5, seed=3)
    nT = len(tets)
    assert nT % 32 and nT % 128  # a partial warp and block
    if squash:  # edges along a coordinate only, and some of no length
        xyz = np.round(xyz, 1)
        xyz[40] = xyz[41]
    c = dict(xyz=xyz, tets=tets, fib=fibres(kind, nT, rng), cf=np.where(np.arange(nT) % 50 < 30, 0.6, 0.5))
    c["ct"] = 0.4 * c["cf"]
    sv, st = np.array([0, 77]), np.array([0.0, 0.4])
    with F.Solver(max_iterations=5000) as s:
        s.set_mesh(xyz, tets)
        s.set_conduction(c["fib"], c["cf"], c["ct"])
        s.set_stimuli(sv, st)
        s.solve()
        phi, state = s.times()
    slots, _, _, _ = O.reference_slots(len(xyz), tets, None)
    geo = O.metric_geo(slots, xyz, c["fib"], c["cf"], c["ct"])
    phi_o, state_o, _, _ = O.solve_pure(len(xyz), slots, geo, sv, st)
    assert np.array_equal(phi, phi_o) and np.array_equal(state, state_o)


@pytest.mark.parametrize("offset", [0, 8, 4], ids=["aligned", "odd double", "odd float"])
def test_device_fields_at_any_address(F, offset):
    import fim_mesh
    torch = pytest.importorskip("torch")
    c = fim_mesh.slab_case(cells=(17, 9, 5), size=(3.4, 1.8, 1.0), scar_radius=0.3, seed=6)
    with F.Solver() as s:
        s.set_mesh(c["xyz"], c["tets"])
        s.set_stimuli(c["seed_v"], c["seed_t"])
        s.set_conduction(c["fib"], c["cf"], c["ct"])
        s.solve()
        phi = s.times(with_state=False)
        keep, ptrs = [], []
        for k in ("fib", "cf", "ct"):
            raw = torch.zeros(c[k].nbytes + 16, dtype=torch.uint8, device="cuda")
            raw[offset:offset + c[k].nbytes] = torch.from_numpy(np.ascontiguousarray(c[k]).view(np.uint8).reshape(-1))
            keep.append(raw)
            ptrs.append(raw.data_ptr() + offset)
        torch.cuda.synchronize()
        X = torch.zeros((len(c["xyz"]), F.MLP_INPUTS), dtype=torch.int16, device="cuda")
        scale = s.features(X.data_ptr())
        s.set_conduction_device(*ptrs)
        keep.clear()  # the field's own memory is not read after the call
        s.solve()
        assert np.array_equal(s.times(with_state=False), phi)
        assert s.features(X.data_ptr()) == pytest.approx(scale, rel=1e-6)
