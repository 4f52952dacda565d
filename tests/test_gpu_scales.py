"""The FP64 triangle solve takes its floats by shifting bit patterns, its
quotient and root from FP32; outside the middle of the float range, on
rounding boundaries and for right angles it falls back.  Meshes scaled far
from 1, and regular grids with isotropic speeds, equal the oracle bit for
bit."""
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


def check(F, O, xyz, tets, fib, cf, ct, sv, st):
    with F.Solver(max_iterations=5000) as s:
        s.set_mesh(xyz, tets)
        s.set_conduction(fib, cf, ct)
        s.set_stimuli(sv, st)
        s.solve()
        phi, state = s.times()
    slots, _, _, _ = O.reference_slots(len(xyz), tets, None)
    geo = O.metric_geo(slots, xyz, fib, cf, ct)
    phi_o, state_o, _, _ = O.solve_pure(len(xyz), slots, geo, sv, st)
    assert np.array_equal(phi, phi_o) and np.array_equal(state, state_o)


# squared lengths from the subnormal floats to the largest
@pytest.mark.parametrize("scale", [1e-22, 1e-20, 1e-18, 1e-12, 1e-6, 1e6, 1e12, 1e18])
@pytest.mark.parametrize("t0", [0.0, 40.0])
def test_scaled_meshes(F, O, scale, t0):
    import fim_mesh
    c = fim_mesh.slab_case(cells=(14, 7, 4), size=(2.8, 1.4, 0.8), scar_radius=0.3, seed=8)
    check(F, O, c["xyz"] * scale, c["tets"], c["fib"], c["cf"], c["ct"], c["seed_v"],
          (c["seed_t"] + t0) * scale)


@pytest.mark.parametrize("n", [4, 9, 16])
def test_regular_grids_with_right_angles(F, O, n):
    import fim_mesh
    c = fim_mesh.cube_case(n, jitter=0.0)
    check(F, O, c["xyz"], c["tets"], c["fib"], c["cf"], c["ct"], c["seed_v"], c["seed_t"])
    # cells of length 1 and unit speeds: sums and roots land on floats
    one = np.ones(len(c["tets"]))
    check(F, O, c["xyz"] * n, c["tets"], c["fib"], one, one, c["seed_v"], c["seed_t"])
