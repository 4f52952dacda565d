"""The learned warm start: the network's GPU kernels against the CPU
restatement (oracle/mlp_oracle.py), training on FIM maps, and warm-started
solves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F(built_library):
    import fim_api
    return fim_api


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _random_problem(M, n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(M.NPARAMS, dtype=np.float32)
    p[M.OW1:M.OW1 + 7 * M.H] = rng.normal(0, 0.5, 7 * M.H)
    p[M.OW2:M.OB1] = rng.normal(0, 0.12, 2 * M.H * M.H)
    p[M.OB1:M.OW4] = rng.normal(0, 0.05, 3 * M.H)
    p[M.OW4:M.OB4] = rng.normal(0, 0.1, M.H)
    p[M.OB4] = 0.3
    X = np.zeros((n, M.IN), dtype=np.float32)
    X[:, :7] = rng.normal(0, 1, (n, 7))
    X = M.bf16(X)
    t = rng.normal(0.5, 0.3, n).astype(np.float32)
    return p, X, t


def _to_device_bf16(torch, X):
    bits = (np.ascontiguousarray(X, dtype=np.float32).view(np.uint32) >> 16).astype(np.uint16)
    return torch.from_numpy(bits.view(np.int16)).cuda()


def test_gradients_match_oracle(F, torch_cuda):
    from oracle import mlp_oracle as M
    torch = torch_cuda
    p, X, t = _random_problem(M, 256, 1)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        assert np.array_equal(mlp.get_params(), p)
        dX, dt = _to_device_bf16(torch, X), torch.from_numpy(t).cuda()
        g, loss = mlp.gradients(256, dX.data_ptr(), dt.data_ptr())
        y = torch.empty(256, dtype=torch.float32, device="cuda")
        mlp.predict(256, dX.data_ptr(), y.data_ptr())
    loss_o, g_o = M.loss_and_gradients(p, X, t)
    _, _, _, y_o = M.forward(p, X)
    assert np.allclose(y.cpu().numpy(), y_o, rtol=1e-3, atol=1e-3)
    assert abs(loss - loss_o) <= 1e-3 * abs(loss_o)
    for name, (a, b) in M.BLOCKS.items():
        ref = g_o[a:b]
        err = np.linalg.norm(g[a:b] - ref) / max(np.linalg.norm(ref), 1e-12)
        assert err < 1e-2, (name, err)


@pytest.mark.parametrize("n", [192, 4096])
def test_tensor_core_gemms_ragged_tile_and_long_k(F, torch_cuda, n):
    """192 rows end in half a 128-row tile (rows past the matrix read as
    zeros and are not stored); 4096 rows make the weight gradients 64 K
    slices, many passes through the GEMM's stage ring."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    p, X, t = _random_problem(M, n, 11)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        dX, dt = _to_device_bf16(torch, X), torch.from_numpy(t).cuda()
        y = torch.empty(n, dtype=torch.float32, device="cuda")
        mlp.predict(n, dX.data_ptr(), y.data_ptr())
        g, loss = mlp.gradients(n, dX.data_ptr(), dt.data_ptr())
        y2 = torch.empty(n, dtype=torch.float32, device="cuda")
        mlp.predict(n, dX.data_ptr(), y2.data_ptr())
    _, _, _, y_o = M.forward(p, X)
    yg = y.cpu().numpy()
    # FP32 summation order differs from the oracle's: where that flips the
    # BF16 rounding of a stored activation, the row moves by a BF16 step
    bad = ~np.isclose(yg, y_o, rtol=1e-3, atol=1e-3)
    assert bad.mean() < 0.01, bad.sum()
    assert np.max(np.abs(yg - y_o)) < 0.05 * np.max(np.abs(y_o))
    assert np.array_equal(yg, y2.cpu().numpy())  # deterministic
    loss_o, g_o = M.loss_and_gradients(p, X, t)
    assert abs(loss - loss_o) <= 1e-3 * abs(loss_o)
    for name, (a, b) in M.BLOCKS.items():
        ref = g_o[a:b]
        err = np.linalg.norm(g[a:b] - ref) / max(np.linalg.norm(ref), 1e-12)
        assert err < 1e-2, (name, err)


def test_row_count_must_be_multiple_of_64(F, torch_cuda):
    torch = torch_cuda
    with F.Mlp() as mlp:
        X = torch.zeros((100, F.MLP_INPUTS), dtype=torch.int16, device="cuda")
        y = torch.zeros(100, dtype=torch.float32, device="cuda")
        with pytest.raises(F.FimError) as e:
            mlp.predict(100, X.data_ptr(), y.data_ptr())
        assert e.value.code == 1


def test_training_beats_the_distance_feature_and_warm_solves(F, torch_cuda):
    """Trained on FIM maps of small slabs, the network predicts held-out maps
    better than the metric distance to the stimuli alone (what it gains over
    the method without it).  A warm-started solve only corrects downwards
    where its start passes the support check; an all-infinite warm start is
    the cold solve bit for bit."""
    import fim_warm
    torch = torch_cuda
    cells = (24, 9, 5)
    train_maps = fim_warm.make_maps(48, cells, 7, torch)
    test_maps = fim_warm.make_maps(6, cells, 8, torch)
    with F.Mlp(seed=5) as mlp:
        losses = fim_warm.train(mlp, train_maps, steps=600, batch=1024, lr=2e-3, torch=torch)
        assert np.mean(losses[-50:]) < 0.3 * np.mean(losses[:10])
        ev = fim_warm.evaluate(mlp, test_maps, torch)
        # measured on the GB300: network RMS error 0.19 of max(t) against 0.30
        # for the distance feature
        assert ev["net_rms"] < 0.8 * ev["dist_rms"], ev
        with F.Solver() as s:
            m = test_maps[0]
            phi, st, start = fim_warm.warm_solve(s, mlp, m, torch)
            other = np.ones(m.nV, dtype=bool)
            other[m.case["seed_v"]] = False
            if st["warm_reset"] == 0:
                assert np.all(phi[other] <= start[other])  # corrections only go down
            assert np.all(phi[m.case["seed_v"]] <= m.case["seed_t"])
            inf = torch.full((m.nV,), float(F.INF), dtype=torch.float64, device="cuda")
            c = m.case
            s.set_mesh(c["xyz"], c["tets"])
            s.set_conduction(c["fib"], c["cf"], c["ct"])
            s.set_stimuli(c["seed_v"], c["seed_t"])
            s.set_warm_start(inf.data_ptr())
            s.solve()
            assert np.array_equal(s.times(with_state=False), m.phi)


@pytest.mark.parametrize("n", [64, 128, 19456 + 64, 77888])
def test_network_tile_counts(F, torch_cuda, n):
    """One half tile, one tile, just over one tile per SM (152 x 128 rows) and
    several tiles per CTA and group: predictions and gradients against the
    restatement, the same bounds as above."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    p, X, t = _random_problem(M, n, 5)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        dX, dt = _to_device_bf16(torch, X), torch.from_numpy(t).cuda()
        y = torch.full((n + 1,), 7.0, dtype=torch.float32, device="cuda")
        mlp.predict(n, dX.data_ptr(), y.data_ptr())
        g, loss = mlp.gradients(n, dX.data_ptr(), dt.data_ptr())
        g2, loss2 = mlp.gradients(n, dX.data_ptr(), dt.data_ptr())
    _, _, _, y_o = M.forward(p, X)
    yg = y.cpu().numpy()
    assert yg[n] == 7.0  # nothing past the rows is written
    assert (~np.isclose(yg[:n], y_o, rtol=1e-3, atol=1e-3)).mean() < 0.01
    assert np.array_equal(g, g2) and loss == loss2  # sums in a fixed order
    loss_o, g_o = M.loss_and_gradients(p, X, t)
    assert abs(loss - loss_o) <= 1e-3 * abs(loss_o)
    for name, (a, b) in M.BLOCKS.items():
        err = np.linalg.norm(g[a:b] - g_o[a:b]) / max(np.linalg.norm(g_o[a:b]), 1e-12)
        assert err < 1e-2, (name, err)


def test_prediction_into_its_own_features_or_an_odd_address(F, torch_cuda):
    """Outputs that the kernel cannot write while it reads (over the feature
    rows) or at all (not aligned to a float) take the copy."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    n = 512
    p, X, _ = _random_problem(M, n, 6)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        dX = _to_device_bf16(torch, X)
        y = torch.empty(n, dtype=torch.float32, device="cuda")
        mlp.predict(n, dX.data_ptr(), y.data_ptr())
        raw = torch.zeros(4 * n + 8, dtype=torch.uint8, device="cuda")
        mlp.predict(n, dX.data_ptr(), raw.data_ptr() + 2)
        odd = raw.cpu().numpy()[2:2 + 4 * n].copy().view(np.float32)
        assert np.array_equal(odd, y.cpu().numpy())
        mlp.predict(n, dX.data_ptr(), dX.data_ptr())
        over = dX.cpu().numpy().reshape(-1)[:2 * n].copy().view(np.float32)
        assert np.array_equal(over, y.cpu().numpy())


@pytest.mark.parametrize("tiles", [153, 304, 305, 456, 457, 761, 3 * 456 + 300])
def test_prediction_rounds_with_few_tiles(F, torch_cuda, tiles):
    """Last rounds in which only some CTAs or only one or two of a CTA's three
    groups have a tile (152 CTAs), the last tile half full: against the
    restatement, the bounds of the other predictions."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    n = 128 * tiles - 64
    p, X, _ = _random_problem(M, n, 7)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        dX = _to_device_bf16(torch, X)
        y = torch.full((n + 1,), 7.0, dtype=torch.float32, device="cuda")
        mlp.predict(n, dX.data_ptr(), y.data_ptr())
    _, _, _, y_o = M.forward(p, X)
    yg = y.cpu().numpy()
    assert yg[n] == 7.0
    assert (~np.isclose(yg[:n], y_o, rtol=1e-3, atol=1e-3)).mean() < 0.01
    assert np.abs(yg[:n] - y_o).max() < 0.05 * np.abs(y_o).max()


@pytest.mark.parametrize("cells,offset", [((1, 1, 1), 0), ((3, 2, 1), 2), ((9, 7, 3), 0), ((9, 7, 3), 6), ((31, 16, 5), 0)])
def test_features_against_their_definition(F, torch_cuda, cells, offset):
    """Every feature from its definition in float64, on a 16-byte boundary and
    off it.  Features are BF16 (relative half step 2^-9; 2^-7 leaves room for
    the FP32 sums before the rounding); the angle and the coordinates lie in
    [-1, 1] and may pass through zero: 2^-8 absolute."""
    import fim_mesh
    torch = torch_cuda
    c = fim_mesh.slab_case(cells=cells, size=(2.0, 1.5, 0.5), seed=11, cf=0.6, ct=0.25, angle=50.0, scar_radius=0.2,
                           n_stim=3, t0_max=5.0)
    xyz, tets = np.asarray(c["xyz"], float), np.asarray(c["tets"])
    nV = xyz.shape[0]
    buf = torch.full((nV * 64 + 16,), 77, dtype=torch.int16, device="cuda")
    with F.Solver() as s:
        s.set_mesh(xyz, tets)
        s.set_conduction(c["fib"], c["cf"], c["ct"])
        s.set_stimuli(c["seed_v"], c["seed_t"])
        scale = s.features(buf.data_ptr() + offset)
    raw = buf.cpu().numpy().view(np.uint16)
    lo = offset // 2
    assert (raw[:lo] == 77).all() and (raw[lo + nV * 64:] == 77).all()
    X = (raw[lo:lo + nV * 64].astype(np.uint32) << 16).view(np.float32).reshape(nV, 64).astype(float)
    sums = np.zeros((nV, 6))
    per_tet = np.column_stack([np.asarray(c["fib"], float), c["cf"], c["ct"], np.ones(len(tets))])
    for k in range(4):
        np.add.at(sums, tets[:, k], per_tet)
    f = sums[:, :3] / np.linalg.norm(sums[:, :3], axis=1, keepdims=True)
    cf, ct = sums[:, 3] / sums[:, 5], sums[:, 4] / sums[:, 5]
    d = xyz[:, None, :] - xyz[np.asarray(c["seed_v"])][None]
    along = np.einsum("vsk,vk->vs", d, f)
    d2 = along ** 2 / cf[:, None] ** 2 + ((d ** 2).sum(-1) - along ** 2) / ct[:, None] ** 2
    dist = (np.asarray(c["seed_t"], float)[None] + np.sqrt(np.maximum(d2, 0))).min(1)
    mid, half = (xyz.max(0) + xyz.min(0)) / 2, (xyz.max(0) - xyz.min(0)) / 2
    assert scale == pytest.approx(dist.max(), rel=1e-5)
    assert np.allclose(X[:, :3], (xyz - mid) / half, rtol=0, atol=2.0 ** -8)
    for k, want in ((3, dist / dist.max()), (4, cf), (5, ct)):
        assert np.allclose(X[:, k], want, rtol=2.0 ** -7, atol=2.0 ** -12), k
    assert np.allclose(X[:, 6], np.arctan2(f[:, 1], f[:, 0]) / np.pi, rtol=0, atol=2.0 ** -8)
    assert (X[:, 7:] == 0).all()


def test_a_refused_training_step_counts_for_nothing(F, torch_cuda):
    """A training step that is refused before anything runs (features off the
    16-byte boundary of the copies) leaves the network as it was, Adam's step
    count included: the next step is the first step's bits."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    n = 128
    p, X, t = _random_problem(M, n, 8)
    dX, dt = _to_device_bf16(torch, np.concatenate([X, X[:1]])), torch.from_numpy(t).cuda()
    got = []
    for refused in (0, 3):
        with F.Mlp(seed=3) as mlp:
            mlp.set_params(p)
            for _ in range(refused):
                with pytest.raises(F.FimError):
                    mlp.train_step(n, dX.data_ptr() + 2, dt.data_ptr(), 1e-2)
                assert np.array_equal(mlp.get_params(), p)
            got.append([(mlp.train_step(n, dX.data_ptr(), dt.data_ptr(), 1e-2), mlp.get_params()) for _ in range(2)])
    for (loss, params), (loss_ref, params_ref) in zip(got[1], got[0]):
        assert loss == loss_ref and np.array_equal(params, params_ref)


def test_a_training_step_whose_wait_ran_out_changes_nothing(F, torch_cuda):
    """With the error words as a CTA whose bounded wait ran out leaves them
    (its sums are missing) the call reports it and parameters, moments and
    step count stay: the steps after it are those of a network without it."""
    import ctypes as C
    from oracle import mlp_oracle as M
    torch = torch_cuda
    n = 512
    p, X, t = _random_problem(M, n, 9)
    dX, dt = _to_device_bf16(torch, X), torch.from_numpy(t).cuda()
    timeout = F.lib().fim_mlp_test_timeout
    timeout.argtypes = [C.c_void_p]
    got = []
    for hit in (False, True):
        with F.Mlp(seed=3) as mlp:
            mlp.set_params(p)
            steps = []
            for i in range(3):
                if hit:
                    before = mlp.get_params()
                    assert timeout(mlp.h) == 0
                    with pytest.raises(F.FimError) as e:
                        mlp.train_step(n, dX.data_ptr(), dt.data_ptr(), 1e-2)
                    assert F.STATUS[e.value.code] == "FIM_ERR_TIMEOUT"
                    assert np.array_equal(mlp.get_params(), before)
                steps.append((mlp.train_step(n, dX.data_ptr(), dt.data_ptr(), 1e-2), mlp.get_params()))
            g, loss = mlp.gradients(n, dX.data_ptr(), dt.data_ptr())
            steps.append((loss, g))
            got.append(steps)
    for (loss, v), (loss_ref, v_ref) in zip(got[1], got[0]):
        assert loss == loss_ref and np.array_equal(v, v_ref)


def test_prediction_into_pinned_host_memory(F, torch_cuda):
    """Outputs that are not on the device take the copy too."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    n = 1024
    p, X, _ = _random_problem(M, n, 10)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        dX = _to_device_bf16(torch, X)
        y = torch.empty(n, dtype=torch.float32, device="cuda")
        h = torch.empty(n, dtype=torch.float32).pin_memory()
        mlp.predict(n, dX.data_ptr(), y.data_ptr())
        mlp.predict(n, dX.data_ptr(), h.data_ptr())
        assert np.array_equal(h.numpy(), y.cpu().numpy())


@pytest.mark.parametrize("tiles", [153, 305, 608, 609])
def test_every_row_of_the_last_tiles(F, torch_cuda, tiles):
    """Tiles in rounds of 304 (two groups of 152 CTAs) or, in training, 152,
    the last one half full: every row's prediction within the bounds of the
    others, twice the same bits, and the gradients of a loss that lies in the
    last tile's rows."""
    from oracle import mlp_oracle as M
    torch = torch_cuda
    n = 128 * tiles - 64
    p, X, _ = _random_problem(M, n, 12)
    _, _, _, y_o = M.forward(p, X)
    t = (y_o + 0.01).astype(np.float32)
    t[-64:] += np.linspace(-30.0, 30.0, 64).astype(np.float32)
    with F.Mlp(seed=3) as mlp:
        mlp.set_params(p)
        dX, dt = _to_device_bf16(torch, X), torch.from_numpy(t).cuda()
        ys = [torch.full((n + 1,), 7.0, dtype=torch.float32, device="cuda") for _ in range(2)]
        for y in ys:
            mlp.predict(n, dX.data_ptr(), y.data_ptr())
        g, loss = mlp.gradients(n, dX.data_ptr(), dt.data_ptr())
    yg = ys[0].cpu().numpy()
    assert yg[n] == 7.0 and np.array_equal(yg, ys[1].cpu().numpy())
    assert np.abs(yg[:n] - y_o).max() < 0.05 * np.abs(y_o).max()
    loss_o, g_o = M.loss_and_gradients(p, X, t)
    assert abs(loss - loss_o) <= 1e-3 * abs(loss_o)
    for name, (a, b) in M.BLOCKS.items():
        err = np.linalg.norm(g[a:b] - g_o[a:b]) / max(np.linalg.norm(g_o[a:b]), 1e-12)
        assert err < 1e-2, (name, err)
