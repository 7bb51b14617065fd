"""Kernel forms at the sizes where they can go wrong: edges of tiles and
stripes, remainders, the smallest and the largest of a form's range.  Each is
held to the oracle, or bit for bit to the general form of the same kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nc", [(1, 1), (2, 5), (3, 3), (5, 1), (9, 33), (40, 31), (64, 32),
                                   (7, 512), (11, 513), (6, 1061)])
@pytest.mark.parametrize("thr", [0.0, 3.0])
def test_hot_pixel_wavefront(capi, oracle, nr, nc, thr):
    """Column stripes of 512 and their remainders; dense outliers (threshold 0,
    and every value below the median), so replacements feed one another."""
    rng = np.random.default_rng(nr * 4099 + nc)
    a = rng.integers(0, 65536, (nr, nc, 2), dtype=np.uint16)
    a[..., 1] = rng.integers(900, 1000, (nr, nc))
    a[rng.random(a.shape) < 0.02] = 65535
    a = np.asfortranarray(a)
    np.testing.assert_array_equal(capi.hot_pixel_filter(a, thr), oracle.hot_pixel_filter(a, thr))


@pytest.mark.parametrize("n", [1, 3, 4, 32, 33, 255, 256, 257, 2500])
def test_mlp_gradient_rows(capi, pkg, oracle, n):
    """Groups of 4 samples, chains of 32 rows, 8 chains at a time and more
    groups than blocks; the tolerances are those of the fixed-size test."""
    import lambda_mlp as lm
    rng = np.random.default_rng(n)
    f = rng.normal(size=(max(n, 2), 67)).astype(np.float32)
    t = rng.uniform(-6, 0, max(n, 2)).astype(np.float32)
    m = pkg.learned.init_model(f, t, seed=n)
    f, t = f[:n], t[:n]
    loss, g = capi.lambda_grad(m, f, t)
    loss0, g0 = lm.loss_and_grad(m, f, t)
    assert abs(loss - loss0) <= 1e-5 * loss0
    assert np.abs(g - g0).max() <= 1e-4 * np.abs(g0).max()
    y0 = lm.predict(m, f)
    assert np.abs(capi.lambda_predict(m, f) - y0).max() <= 1e-4 * (1 + np.abs(y0).max())


@pytest.mark.parametrize("n", [480, 512, 513, 1024, 1025, 9000, 65536, 65537, 131105])
def test_mlp_gradient_of_many_rows(capi, pkg, oracle, n):
    """Either side of the number of rows from which the chains have a kernel of
    their own, full and cut last chains, one to three slabs of chains; the tolerances
    are those of the fixed-size test."""
    test_mlp_gradient_rows(capi, pkg, oracle, n)


def _noisy(pkg, side, nt, seed):
    return pkg.synth.workload("arps_256", seed=seed, side=side, nt=nt)


@pytest.mark.parametrize("bs,T", [(2, 3), (3, 7), (4, 9), (4, 11), (4, 15)])
@pytest.mark.parametrize("expw", [0, 1])
def test_sorted_factors_are_identical(capi, pkg, bs, T, expw):
    """The two-kernel SVD form (columns sorted by the sweeps, factors of four
    triplets at a time) against the shared-memory form, bit for bit; without
    exponential weighting every triplet survives, more than four."""
    noisy, _, (a, m, s) = _noisy(pkg, 37, T + 3, 40 + bs)
    out = []
    for form in (0, 3):
        p = capi.default_params(traj_length=T, block_size=bs, motion_window=5, median_size=-1,
                                random_seed=3, alpha=a / 300, mu=m / 300, sigma=s / 300,
                                exp_weighting=expw, autotune=form)
        Y, est, _, ex = capi.denoise_ex(noisy, p)
        out.append((Y, est, ex["risk"]))
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("bs,T", [(5, 7), (6, 9), (7, 11), (8, 15)])
def test_qr_factors_of_every_triplet(capi, pkg, oracle, bs, T):
    """More surviving triplets than the QR form's factors take at a time, against
    the oracle at a fixed threshold (the whole-sequence tolerance at fixed
    lambda)."""
    noisy, _, _ = _noisy(pkg, 33, T + 2, 50 + bs)
    kw = dict(traj_length=T, block_size=bs, motion_window=5, median_size=-1, random_seed=3,
              optimize_pgure=0, exp_weighting=0, lambda_=0.002)
    Y, _, _ = capi.denoise(noisy, capi.default_params(autotune=5, **kw))
    Yo, _, _ = oracle.denoise(noisy, n_jobs=4, **kw)
    assert np.abs(Y - Yo).max() <= 2e-5 * np.abs(Yo).max()


@pytest.mark.parametrize("bs,T,side", [(2, 3, 21), (3, 7, 30), (4, 15, 35), (5, 9, 29), (6, 21, 31),
                                       (7, 15, 26), (8, 21, 33), (9, 9, 30), (16, 21, 40)])
@pytest.mark.parametrize("nl", [1, 2, 9, 16])
def test_eval_round_of_any_length(capi, pkg, oracle, bs, T, side, nl):
    """Rounds of one to sixteen lambda values (single, paired, odd; the smaller
    tiles of long rounds), every patch side's rows per pass, against the
    oracle's risks (the tolerance of the risk tests)."""
    noisy, _, _ = _noisy(pkg, side, T + 2, 60 + bs)
    lams = np.geomspace(0.01, 20.0, nl)
    noise = dict(alpha=0.01, mu=0.02, sigma=0.03)
    p = capi.default_params(traj_length=T, block_size=bs, motion_window=5, median_size=-1,
                            random_seed=3, **noise)
    res, _ = capi.denoise_batch([dict(X=noisy, params=p, lambdas=lams)])
    fw = min(T, bs * bs - 1) // 2
    u = np.asarray(noisy[..., :2 * fw + 1], np.float64)
    u = u / u.max()
    rows, cols = oracle.arps_window(u, bs, 5, fw, fw, T + 2)
    ro = oracle.risk_window(u, bs, 1, rows, cols, lams, *noise.values(), 3)
    r = res[0]["risks"][fw]
    assert np.abs(r - ro).max() <= 1e-4 * np.abs(ro).max()


@pytest.mark.parametrize("bs,T", [(5, 7), (5, 15), (6, 21), (7, 9), (7, 21), (8, 21)])
@pytest.mark.parametrize("expw", [0, 1])
def test_owner_forms_are_identical(capi, pkg, bs, T, expw):
    """The register forms whose pairs are owned by one of 8 or 16 lanes (one or
    two pairs each) against the shared-memory form, whose rotations every lane
    computes: bit for bit."""
    noisy, _, (a, m, s) = _noisy(pkg, 31, T + 2, 70 + bs)
    out = []
    for form in (0, 3):
        p = capi.default_params(traj_length=T, block_size=bs, motion_window=5, median_size=-1,
                                random_seed=3, alpha=a / 300, mu=m / 300, sigma=s / 300,
                                exp_weighting=expw, autotune=form)
        if form == 0 and bs >= 7 and T <= 15:
            p.autotune = 5  # the QR form is the default there; compare it loosely
        Y, est, st, ex = capi.denoise_ex(noisy, p)
        out.append((Y, est, ex["risk"], st.svd_variant))
    if out[0][3] == 4:
        assert np.abs(out[0][0] - out[1][0]).max() <= 2e-5 * np.abs(out[1][0]).max()
        return
    for x, y in zip(out[0][:3], out[1][:3]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("points", [9, 10, 11, 12, 13, 16])
@pytest.mark.parametrize("bs,T", [(3, 7), (4, 9), (4, 13), (4, 15)])
@pytest.mark.parametrize("mode", ["plain", "hint", "learned", "budget"])
def test_rounds_shorter_than_the_grid(capi, pkg, oracle, points, bs, T, mode):
    """Searches of 9 to 16 grid points whose later rounds hold fewer values than
    their launch allocates for: refinements of half the points, narrow searches of
    4 to 6, a budget of 8 evaluations.  Against the oracle's risk at the returned
    lambda (the tolerance of the risk tests), and its own search from the same
    proposals (that of the search tests)."""
    noisy, _, _ = _noisy(pkg, 32, T + 1, 80 + bs)
    X = noisy.astype(np.float64)
    fw = min(T, bs * bs - 1) // 2
    noise = dict(alpha=0.01, mu=0.02, sigma=0.03)
    kw = dict(traj_length=T, block_size=bs, motion_window=5, median_size=-1, random_seed=3,
              search_points=points, frame_begin=fw, frame_end=fw + 1, **noise)
    hints = None
    if mode == "hint":
        kw["lambda_hint"] = 1.0
    elif mode == "budget":
        kw["max_iter"] = 8
    elif mode == "learned":
        model = pkg.learned.load_model()
        kw["lambda_model"] = model.ctypes.data
    _, est, _, ex = capi.denoise_ex(X, capi.default_params(**kw), proposals=True)
    if mode == "learned":
        kw.pop("lambda_model")
        hints = 100.0 * 10.0 ** np.clip(ex["proposals"].astype(np.float64), -6, 0)
        hints = np.nan_to_num(hints, nan=1.0)  # frames out of range have no proposal
    _, est0, rep = oracle.denoise(X, lambda_hints=hints, n_jobs=4, **kw)
    u = X[:, :, :2 * fw + 1] / X[:, :, :2 * fw + 1].max()
    rows, cols = oracle.arps_window(u, bs, 5, fw, fw, T + 1)
    r = oracle.risk_window(u, bs, 1, rows, cols, [est[fw, 0], est0[fw, 0]], *noise.values(), 3)
    assert abs(ex["risk"][fw] - r[0]) <= 1e-4 * abs(r[0])
    assert (r[0] - r[1]) / abs(r[1]) < 0.01
    if mode == "budget":
        assert ex["evals"][fw] <= 8


@pytest.mark.parametrize("side,nwin", [(8, 3), (17, 5), (21, 15), (32, 15)])
@pytest.mark.parametrize("seed", [0, 11, 2 ** 63 - 1])
def test_probe_streams(capi, oracle, side, nwin, seed):
    """The probes are drawn on the device, 16 draws per thread: window sizes that
    are and are not multiples of 16, both probe sets (without the integer-delta1
    quirk the risk depends on delta1 as well), against the oracle's risk (the
    tolerance of the risk tests)."""
    rng = np.random.default_rng(side + nwin)
    u = rng.uniform(0.2, 1.0, (side, side, nwin))
    u /= u.max()
    P = (side - 4 + 1) ** 2
    rows = np.tile(np.arange(P) % (side - 3), (nwin, 1)).astype(np.int32)
    cols = np.tile(np.arange(P) // (side - 3), (nwin, 1)).astype(np.int32)
    for compat in (capi.COMPAT_ALL, capi.COMPAT_ALL & ~capi.COMPAT_INT_DELTA1):
        args = (u, 4, 1, rows, cols, [0.5, 5.0], 0.02, 0.03, 0.05, seed, compat)
        r, ro = capi.risk_window(*args), oracle.risk_window(*args)
        assert np.abs(r - ro).max() <= 1e-4 * np.abs(ro).max()


@pytest.mark.parametrize("bs,vmax,dtype", [(4, 1023, "uint16"), (4, 1025, "uint16"), (8, 511, "uint16"),
                                           (8, 513, "float32"), (9, 65535, "uint16"), (2, 2047, "uint16"),
                                           (5, 524288, "float32"), (4, 524289, "float32"),
                                           (3, 3, "uint8"), (6, 7, "uint8")])
def test_arps_cost_forms(capi, oracle, bs, vmax, dtype):
    """Exact FP32 sums up to m * max^2 = 2^24, 64-bit ones to values of 2^19, FP32
    with error bounds beyond; few grey levels give many ties.  Motion vectors are
    those of the oracle, so the output is too (the whole-sequence tolerance at
    fixed lambda)."""
    rng = np.random.default_rng(bs * 1000 + vmax % 97)
    side, T = 34, 7 if bs > 2 else 3
    base = rng.integers(0, vmax + 1, (side + 8, side + 8))
    base[::3] = vmax
    X = np.stack([base[2 + k % 3:2 + k % 3 + side, 4 - k % 4:4 - k % 4 + side] for k in range(T + 1)], -1)
    X = np.asfortranarray(X.astype(dtype))
    kw = dict(traj_length=T, block_size=bs, motion_window=7, median_size=-1, random_seed=3,
              optimize_pgure=0, lambda_=0.05)
    Y, _, _ = capi.denoise(X, capi.default_params(**kw))
    Yo, _, _ = oracle.denoise(X, n_jobs=4, **kw)
    assert np.abs(Y - Yo).max() <= 2e-5 * np.abs(Yo).max()


def _noise_window(kind, side, T):
    """Frames of the noise estimator's rare cases, maximum 1."""
    rng = np.random.default_rng(side + T)
    if kind == "random":
        u = 1.0 + rng.random((side, side, 1)) * rng.random((side, side, T))
    else:
        # three quarters made of one 8 x 8 tile each: a few hundred equal leaves
        u = 1.0 + 0.3 * rng.random((side, side, T))
        y, x = np.mgrid[0:8, 0:8] / 7.0
        h = side // 2
        for q, (r, c) in enumerate(((0, 0), (0, h), (h, 0))):
            tile = 0.5 + 0.7 * q + (x + q * y) ** 2 + 0.05 * (q + 1) * rng.random((8, 8))
            u[r:r + h, c:c + h] = np.tile(tile, (h // 8, h // 8))[:, :, None]
    return np.asfortranarray(u / u.max())


@pytest.mark.parametrize("kind,side,T", [("random", 16, 5), ("random", 32, 15), ("random", 128, 5),
                                         ("tiles", 64, 7), ("tiles", 256, 5)])
def test_noise_estimates_of_equal_and_few_leaves(capi, oracle, kind, side, T):
    """Frames of one to a thousand leaves; equal leaves have equal residuals,
    which the bracketed order statistics must hand to the radix selection.
    1e-4: the robust means stop on an absolute tolerance of 1e-6."""
    u = _noise_window(kind, side, T)
    for method in (1, 2, 3, 4):
        p = capi.default_params(median_size=0, traj_length=T, noise_method=method, random_seed=3,
                                search_points=4, search_rounds=1)
        _, est, _ = capi.denoise(u, p)
        ref = oracle.noise_estimate(u, method=method)
        np.testing.assert_allclose(est[:, 1:], np.tile(ref, (T, 1)), rtol=1e-4)


def test_risk_window_without_lambdas(capi, oracle):
    """No lambda value: an empty result, and nothing of the call is left running on
    memory that the next call gets (its results are those of a call before)."""
    rng = np.random.default_rng(5)
    u = rng.uniform(0.2, 1.0, (64, 64, 15))
    u /= u.max()
    P = 61 * 61
    rows = np.tile(np.arange(P) % 61, (15, 1)).astype(np.int32)
    cols = np.tile(np.arange(P) // 61, (15, 1)).astype(np.int32)
    args = (0.02, 0.03, 0.05, 7)
    r0 = capi.risk_window(u, 4, 1, rows, cols, [0.5, 5.0], *args)
    ro = oracle.risk_window(u, 4, 1, rows, cols, [0.5, 5.0], *args)
    assert np.abs(r0 - ro).max() <= 1e-4 * np.abs(ro).max()
    for _ in range(8):
        assert capi.risk_window(u, 4, 1, rows, cols, [], *args).size == 0
        np.testing.assert_array_equal(capi.risk_window(u, 4, 1, rows, cols, [0.5, 5.0], *args), r0)
    with pytest.raises(RuntimeError):  # the other arguments are still checked
        capi.risk_window(u, 4, 1, rows + 61, cols, [], *args)


@pytest.mark.parametrize("side,flat", [(32, 403.0), (32, 777.0), (32, 835.0), (32, 3943.0),
                                       (64, 835.0), (128, 3943.0)])
def test_flat_blocks_are_not_split(capi, oracle, side, flat):
    """A quadrant of one value: its variance and its residuals' variance are both
    zero, which is no split.  The values are chosen so that flat / sqrt(30) in FP64
    ends in zero bits enough for the quadrant's residuals to add up exactly in any
    order (and the maximum is a power of two, so that the oracle's normalised frames
    behave the same): a residual off by one rounding makes the block split, which
    changes the estimates by a tenth to a factor of three."""
    rng = np.random.default_rng(1)
    h = side // 2
    y, x = np.mgrid[0:side, 0:side] * 32.0 / side
    u = rng.poisson(200 + 20 * x + 9 * y, (3, side, side)).astype(np.float64).transpose(1, 2, 0)
    u = np.minimum(u, 4000.0)
    u[h:, h:] = flat
    u[0, 0] = 4096.0
    u = np.asfortranarray(u)
    res = flat / np.sqrt(30.0)
    assert (np.cumsum(np.full(h * h, res)) == np.arange(1, h * h + 1) * res).all()
    for method in (1, 2, 3, 4):
        p = capi.default_params(median_size=0, traj_length=3, noise_method=method, random_seed=3,
                                search_points=4, search_rounds=1)
        _, est, _ = capi.denoise(u, p)
        ref = oracle.noise_estimate(u / 4096.0, method=method)
        np.testing.assert_allclose(est[:, 1:], np.tile(ref, (3, 1)), rtol=1e-4)


@pytest.mark.parametrize("side", [1024, 2048])
def test_noise_of_large_frames(capi, oracle, side):
    """The largest frames whose quadtree nodes stay in shared memory, and frames
    whose nodes do not; every level splits somewhere."""
    rng = np.random.default_rng(side)
    y, x = np.mgrid[0:side, 0:side] / side
    u = rng.poisson(50 + 40 * np.sin(9 * x) * np.cos(7 * y)) + rng.normal(0, 3, (side, side))
    u = np.maximum(u, 0.0)[:, :, None]
    u = np.asfortranarray(u / u.max())
    p = capi.default_params(median_size=0, traj_length=1, random_seed=3, search_points=4,
                            search_rounds=1)
    _, est, _ = capi.denoise(u, p)
    np.testing.assert_allclose(est[0, 1:], oracle.noise_estimate(u), rtol=1e-4)


def test_fresh_probes_of_every_window(capi, pkg):
    """A negative seed draws new probes for each window of a batch.  On equal windows
    one shared set gives equal risks; fresh sets give risks that all differ, spread
    as those of 24 seeds are (7 windows: within a factor of 10 of their deviation, and
    6 deviations of their mean)."""
    noisy, _, _ = _noisy(pkg, 32, 1, 91)
    X = np.asfortranarray(np.repeat(noisy[:, :, :1], 13, axis=2))
    kw = dict(traj_length=7, motion_window=5, median_size=-1, alpha=0.01, mu=0.02, sigma=0.03,
              window_batch=4)

    def risks(seed, **more):
        p = capi.default_params(random_seed=seed, **kw, **more)
        res, _ = capi.denoise_batch([dict(X=X, params=p, lambdas=[1.0])])
        return res[0]["risks"][3:10, 0]

    seeded = []
    for seed in range(24):
        r = risks(seed)
        assert (r == r[0]).all()
        seeded.append(r[0])
    m, sd = np.mean(seeded), np.std(seeded)
    assert sd > 0 and len(set(seeded)) == 24
    for compat in (capi.COMPAT_ALL, capi.COMPAT_ALL & ~capi.COMPAT_INT_DELTA1):
        r = risks(-1, compat_flags=compat)
        assert len(set(r)) == 7  # windows of three batches
        if compat == capi.COMPAT_ALL:
            assert np.abs(r - m).max() < 6 * sd
            assert sd / 10 < np.std(r) < 10 * sd
    assert set(risks(-1)) != set(risks(-1))


def _saturated(kind, side, nt):
    """Byte frames with clipped highlights, or flat 16 x 16 tiles in noise: patches
    whose columns are equal in many frames."""
    rng = np.random.default_rng(side + nt)
    y, x = np.mgrid[0:side, 0:side]
    f = []
    for k in range(nt):
        b = 40 + 30 * np.sin((x + k) / 5.0) * np.cos((y - k) / 7.0)
        v = (np.minimum(rng.poisson(2 * b), 90) if kind == "clipped" else
             np.where((x // 16 + 2 * (y // 16) + k) % 3 == 0, 3.0 + (x // 16) * 7 + k, rng.poisson(b)))
        f.append(v)
    return np.asfortranarray(np.stack(f, -1).astype(np.uint8))


@pytest.mark.parametrize("bs,T,form", [(4, 15, 0), (4, 9, 3), (5, 9, 0), (5, 9, 5), (6, 15, 5),
                                       (7, 7, 0), (8, 9, 0), (8, 15, 3), (8, 21, 0)])
@pytest.mark.parametrize("kind", ["clipped", "flat"])
@pytest.mark.parametrize("lam,expw", [(0.49, 0), (0.01, 0), (1e-4, 0), (1e-7, 0), (0.0, 0), (0.3, 1)])
def test_patches_of_equal_columns(capi, oracle, kind, bs, T, form, lam, expw):
    """Each equal column leaves 1e-7 of the norm in the QR form, so the fourth has
    a squared norm that FP32 cannot invert; and singular values of rounding noise,
    which a threshold near 0 keeps.  Every form against the oracle at a fixed
    threshold (the whole-sequence tolerance at fixed lambda)."""
    X = _saturated(kind, 64, T)
    kw = dict(traj_length=T, block_size=bs, block_overlap=2, motion_window=3, median_size=-1,
              random_seed=11, optimize_pgure=0, exp_weighting=expw, lambda_=lam)
    Y, _, _ = capi.denoise(X, capi.default_params(autotune=form, frame_begin=2, frame_end=4, **kw))
    Yo, _, _ = oracle.denoise(X, n_jobs=8, frame_begin=2, frame_end=4, **kw)
    assert np.abs(Y - Yo).max() <= 2e-5 * np.abs(Yo).max()
