"""The digit-slice E-step, responsibility pass, map and critical temperature where
values or responsibilities span many powers of two, against the oracle, point by
point and centre by centre."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [3.0, 1.04])  # mantissas of c log2 e just above and well above a power of two
def test_far_centre_beyond_512_bits(pkg, orc, c):
    """A centre whose responsibilities are 2^-600 .. 2^-950: FP64 holds them, so its G,
    RT and R are those of the oracle and its critical temperature is finite."""
    rng = np.random.default_rng(4)
    N, D, K, temp, eps = 3000, 40, 30, 1.1, 1e-6
    s = 0.2 / np.sqrt(c)
    T = s * rng.normal(size=(N, D))
    Y = s * rng.normal(size=(K, D))
    beta = 2.0 * temp * c
    Y[9] = 0.0
    Y[9, 0] = np.sqrt(2.0 * 640.0 / beta) + 0.5
    R, _, _ = orc.resp(orc.dist(Y, T), beta, 1, temp)
    assert 0.0 < R[9].max() < 2.0 ** -560
    with pkg.Context(T, np.ones((K, 1)), "fp64") as ctx:
        assert ctx.path == "exact_slices"
        ctx.set_Y(Y)
        ctx.estep(beta, 1, temp)
        Rb = ctx.R_block(9, 1, 0, N)[0]
        got, got_k = ctx.next_ctemp(temp, beta, eps, per_centre=True)
        ctx.mstep()
        G, RT = ctx.get_stats()
    # the oracle's exp(-beta d / 2) is subnormal, and short of bits, from 708 on
    normal = 0.5 * beta * orc.dist(Y[9:10], T)[0] < 708.0
    assert normal.sum() > 2000
    # an exponent of 600 nats carries 600 x 2^-53 x a few
    assert np.max(np.abs(Rb[normal] / R[9][normal] - 1.0)) <= 1e-11
    gk = R[9].sum()
    assert G[9] == pytest.approx(gk, rel=1e-11)
    assert np.max(np.abs(RT[9] - R[9] @ T)) <= 1e-11 * np.max(np.abs(R[9] @ T))
    assert np.isfinite(got_k[9]) and np.isfinite(got) and got == np.max(got_k)


def test_switch_keeps_the_normal_equations_on_the_cuda_cores(pkg, monkeypatch):
    """DGTM_X64=0 is the arm without digit slices: also for A = FI^T diag(G) FI, whose
    slices take eight launches (the chain's two among them) instead of two."""
    rng = np.random.default_rng(8)
    K, M1, D = 8000, 65, 166
    T = rng.random((260, D))
    FI = np.concatenate([rng.random((K, M1 - 1)), np.ones((K, 1))], axis=1)
    Y = rng.random((K, D))
    launches, W = [], []
    for on in ("1", "0"):
        monkeypatch.setenv("DGTM_X64", on)
        with pkg.Context(T, FI, "fp64") as c:
            assert (c.path == "cuda_cores") == (on == "0")
            c.set_timing(True)
            c.set_Y(Y)
            c.estep(2.0, 1, 1.5)
            W.append(c.mstep()[1])
            G, RT = c.get_stats()
            launches.append(c.timing()["mstep_solve"]["launches"])
    # the reduction of the CUDA-core responsibility pass is one launch more there
    assert launches[0] == launches[1] - 1 + 6
    tol = 16 * M1 * np.finfo(float).eps * np.linalg.cond(FI.T @ (G[:, None] * FI))
    assert np.linalg.norm(W[0] - W[1]) <= tol * np.linalg.norm(W[1])


@pytest.mark.parametrize("pairs", ["1", "0"])
@pytest.mark.parametrize("c", [3.0, 1.04])
def test_critical_temperature_of_a_far_centre(pkg, orc, monkeypatch, pairs, c):
    """The squares of a scatter matrix that follows R = 2^-850 are outside FP64: the
    eigenvalue step still finds its eigenvalues, from both scatters."""
    monkeypatch.setenv("DGTM_CTEMP_PAIRS", pairs)
    rng = np.random.default_rng(4)
    N, D, K, temp, eps = 3000, 40, 30, 1.1, 1e-6
    s = 0.2 / np.sqrt(c)
    T = s * rng.normal(size=(N, D))
    Y = s * rng.normal(size=(K, D))
    beta = 2.0 * temp * c
    Y[9] = 0.0
    Y[9, 0] = np.sqrt(2.0 * 640.0 / beta) + 0.5
    R, _, _ = orc.resp(orc.dist(Y, T), beta, 1, temp)
    with pkg.Context(T, np.ones((K, 1)), "fp64") as ctx:
        ctx.set_Y(Y)
        ctx.estep(beta, 1, temp)
        got_k = ctx.next_ctemp(temp, beta, eps, per_centre=True)[1]
    X = T - Y[9]
    lam = np.linalg.eigvalsh((X * (R[9] / R[9].sum())[:, None]).T @ X * 2.0)  # R^2 is below FP64's range
    lam[lam >= (temp - eps) * 2.0 / beta] = 0.0
    # 2^-53 of the largest eigenvalue, which is 1600 times this one
    assert got_k[9] == pytest.approx(beta / 2.0 * lam.max(), rel=1e-10)


def outlier_case(value, D, own, seed=5, N=1000, K=400):
    """Unit-sized data with one coordinate of one point replaced; own: centre 7 sits on
    that point."""
    rng = np.random.default_rng(seed)
    means = rng.random((16, D))
    T = means[rng.integers(0, 16, N)] + 0.2 * rng.normal(size=(N, D))
    Y = T[rng.integers(0, N, K)] + 0.1 * rng.normal(size=(K, D))
    T[5, D // 2] = value
    if own:
        Y[7] = T[5]
    return T, Y, rng.normal(size=(K, 2))


OUTLIERS = [(v, D, own) for v in (1e3, 1e6, 1e30) for D in (2, 5, 12, 70) for own in (False, True)]


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("value,D,own", OUTLIERS)
def test_one_large_value_leaves_the_other_points_alone(pkg, orc, value, D, own, form):
    """R and the map of every other point, at the bounds that hold without the value:
    1e-13 on R, 1e-12 on the map (FP64 form; the FP32 form's statistics are FP32, and
    one large centre or point does not make them worse)."""
    N, K = (1000, 400) if form == "fp64" else (8000, 300)  # the FP32 form's map by slices
    T, Y, X = outlier_case(value, D, own, N=N, K=K)
    beta, temp = 60.0 * 12 / max(D, 12), 1.5
    with np.errstate(over="ignore", invalid="ignore"):
        R, _, _ = orc.resp(orc.dist(Y, T), beta, 1, temp)
    others = np.arange(N) != 5
    with pkg.Context(T, np.ones((K, 1)), form) as c:
        c.set_Y(Y)
        c.estep(beta, 1, temp)
        M = c.map(X)
        Rb = c.R_block(0, K, 0, N)
    if form == "fp64":
        assert np.max(np.abs(Rb - R)[:, others]) <= 1e-13
        assert np.max(np.abs((M - R.T @ X)[others])) <= 1e-12 * np.max(np.abs(X))
    else:
        assert np.max(np.abs(Rb - R)[:, others]) <= 1e-3
        assert np.max(np.abs((M - R.T @ X)[others])) <= 1e-3 * np.max(np.abs(X))
    # the point itself: its own centre's, or (every exp(-beta d / 2) is 0) any centre's.
    # (Its FP32 distance of 1e6 - 1e6 says nothing; |t|^2 = 1e60 is too much for FP64 too.)
    if (form == "fp64" and value < 1e30) or not own:
        assert np.max(np.abs(Rb[:, 5] - (np.eye(K)[7] if own else 1.0 / K))) <= 1e-13


@pytest.mark.parametrize("value,D,where", [(v, D, w) for v in (1e3, 1e6, 1e30) for D in (5, 12, 70)
                                           for w in ("point", "centre", "both") if not (w == "both" and v == 1e30)])
def test_one_large_value_leaves_the_statistics_alone(pkg, orc, value, D, where):
    """G and R T centre by centre and column by column, 1e-12 of the sum of magnitudes, with
    a far point (the CUDA-core kernels), a far centre (the slices) and a centre on the far
    point."""
    N, K = 1000, 400
    T, Y, _ = outlier_case(value if where != "centre" else 0.5, D, where == "both")
    if where == "centre":
        Y[7, D // 2] = value
    beta, temp = 60.0 * 12 / max(D, 12), 1.5
    with np.errstate(over="ignore", invalid="ignore"):
        R, _, _ = orc.resp(orc.dist(Y, T), beta, 1, temp)
    with pkg.Context(T, np.ones((K, 1)), "fp64") as c:
        assert c.path == ("exact_slices" if where == "centre" else "cuda_cores")
        c.set_Y(Y)
        c.estep(beta, 1, temp)
        c.mstep()
        G, RT = c.get_stats()
    assert np.max(np.abs(G - R.sum(1)) / np.maximum(R.sum(1), 1e-300)) <= 1e-12
    assert np.max(np.abs(RT - R @ T) / np.maximum(R @ np.abs(T), 1e-300)) <= 1e-12


@pytest.mark.parametrize("kind,slices", [("gauss", True), ("uniform", True), ("sparse", True), ("offset", True),
                                         ("outlier", False), ("lognormal", False)])
def test_which_columns_keep_the_digit_slices(pkg, kind, slices):
    """The rule on the columns: ordinary and exactly held data keep the slices."""
    rng = np.random.default_rng(6)
    N, D, K = 4000, 20, 100
    T = rng.normal(size=(N, D))
    if kind == "uniform":
        T = rng.random((N, D))
    elif kind == "sparse":  # mostly zeros, and values of few bits
        T = (rng.random((N, D)) < 0.02) * rng.integers(1, 1000, (N, D)).astype(float)
    elif kind == "offset":
        T += 1e6
    elif kind == "outlier":
        T[17, 3] = 200.0
    elif kind == "lognormal":
        T[:, 4] = np.exp(2.0 * T[:, 4])
    with pkg.Context(T, np.ones((K, 1)), "fp64") as c:
        assert (c.path == "exact_slices") == slices


def test_scatter_with_one_value_far_from_the_mean(pkg, monkeypatch):
    """A column around 1000 with one value of 30,000, which has a centre of its own, fits its
    grid as data, but the squares about the mean do not: the other centres go through the
    CUDA-core scatter.  (2^-57 of the square's grid is 4e-9 a point; the distances' own
    1e6 2^-53 is 1e-10.)"""
    rng = np.random.default_rng(12)
    N, D, K = 6000, 20, 60
    T = rng.normal(size=(N, D))
    T[:, 0] += 1000.0
    Y = T[rng.integers(0, N, K)] + 0.5 * rng.normal(size=(K, D))
    T[11, 0] = 30000.0
    Y[7] = T[11]
    beta = 0.3
    out = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DGTM_CTEMP_PAIRS", pairs)
        with pkg.Context(T, np.ones((K, 1)), "fp64") as c:
            assert c.path == "exact_slices"
            c.set_Y(Y)
            c.estep(beta, 1, 2.0)
            out.append(c.next_ctemp(50.0, beta, 1e-6, per_centre=True)[1])
            R = c.R_block(0, K, 0, N)
    # 8 bits of 2^-53 of the trace may go
    trace = np.array([(R[k][:, None] * (T - Y[k]) ** 2).sum() for k in range(K)]) / R.sum(1)
    assert np.median(trace) < 100.0
    assert np.all(np.abs(out[0] - out[1]) <= 1e-13 * out[1] + 2.0 ** -45 * beta * trace)


def long_double_solve(FI, G, RT):
    """FI W = Y of the normal equations, Cholesky in long double."""
    F = FI.astype(np.longdouble)
    A, B = F.T @ (G.astype(np.longdouble)[:, None] * F), F.T @ RT.astype(np.longdouble)
    n = len(A)
    L = np.zeros_like(A)
    for j in range(n):
        v = A[j:, j] - L[j:, :j] @ L[j, :j]
        L[j:, j] = v / np.sqrt(v[0])
    y = np.zeros_like(B)
    for j in range(n):
        y[j] = (B[j] - L[j, :j] @ y[:j]) / L[j, j]
    w = np.zeros_like(y)
    for j in range(n - 1, -1, -1):
        w[j] = (y[j] - L[j + 1:, j] @ w[j + 1:]) / L[j, j]
    return F @ w


@pytest.mark.parametrize("decades", [0.0, 2.0, 8.0, 12.0])
def test_normal_equations_where_the_weights_span_decades(pkg, monkeypatch, decades):
    """G falls over the map: the centres' error against long double is no larger than with
    the multiply-add chain (a factor of 4 for chance; the slices alone are 100 to 1000
    times the chain at 8 and 12 decades)."""
    K, D = 8000, 8
    x = np.stack(np.meshgrid(*[np.linspace(-1.0, 1.0, 20)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    mu = np.stack(np.meshgrid(*[np.linspace(-4 / 3, 4 / 3, 4)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    e = np.exp(((x[:, None, :] - mu[None]) ** 2).sum(2) * (-0.5 / (4 / 9) ** 2))
    FI = np.concatenate([e, np.ones((K, 1))], axis=1)
    rng = np.random.default_rng(9)
    # all points at one end of a line of centres: R falls as exp(-c d)
    T = 0.05 * rng.normal(size=(400, D)) + 0.5
    Y = T[0] + 0.02 * rng.normal(size=(K, D))
    Y[:, 0] += x[:, 0] + 1.0
    c = decades * np.log(10.0) / 4.0
    beta, temp = max(2.0 * c, 1e-3), 1.0
    err = []
    for on in ("1", "0"):
        monkeypatch.setenv("DGTM_X64", on)
        with pkg.Context(T, FI, "fp64") as ctx:
            ctx.set_Y(Y)
            ctx.estep(beta, 1, temp)
            Yn = ctx.mstep(want_Y=True)[2]
            G, RT = ctx.get_stats()
        if decades:
            assert 0.5 * decades < np.log10(G.max() / G.min()) < 1.6 * decades
        err.append(float(np.max(np.abs(Yn - long_double_solve(FI, G, RT)))))
    assert err[0] <= 4.0 * err[1]


@pytest.mark.parametrize("D,limit", [(5, 400), (9, 800), (37, 2200)])
def test_memory_of_a_context_per_point(pkg, D, limit):
    """Digit planes take what D needs (16 bytes of a value rounded up to 8, twice), not
    whole panels of 64: bytes a point, from contexts of two sizes."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    T = rng.random((2_000_000, D))
    used = []
    for N in (1_000_000, 2_000_000):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with pkg.Context(T[:N], np.ones((64, 1)), "fp64") as c:
            assert c.path == "exact_slices"
            used.append(before - torch.cuda.mem_get_info()[0])
    assert (used[1] - used[0]) / 1e6 <= limit


def test_sums_that_few_points_carry(pkg):
    """Centres of 5000 points whose G lies on a few points each: a unit that 5000 full
    terms would need is 2^-49 of the grids (1e-14 of G here); the sums' own rounding is
    2^-53."""
    rng = np.random.default_rng(15)
    N, D, K = 5000, 9, 1000
    T = rng.random((N, D)) + 0.5
    Y = np.full((K, D), 40.0)  # far from all, but
    Y[:N // 50] = T[:N // 50]  # on the first points
    with pkg.Context(T, np.ones((K, 1)), "fp64") as c:
        assert c.path == "exact_slices"
        c.set_Y(Y)
        c.estep(4000.0, 1, 1.0)
        R = c.R_block(0, N // 50, 0, N)
        c.mstep()
        G, _ = c.get_stats()
    g = R.sum(1, dtype=np.longdouble)
    # 2^-53 each from the block's R and from G's rounding, and half a unit of R's digits
    # (2^-55 of a grid that ends below 4.2 Rmax) from each of a few points
    assert np.max(np.abs(G[:N // 50] / g - 1.0)) <= 2.0 ** -51


def test_scatter_where_few_points_carry_a_centre(pkg, monkeypatch):
    """5001 points and centres whose R lies on a few dozen: the products' sums are rounded
    where they are, not on a unit that 5001 full terms would need (2^-49 of the grids:
    1e-12 of a critical temperature).  8 bits of 2^-53 may go to the expansion, 2.8e-14 of
    the largest eigenvalue."""
    rng = np.random.default_rng(14)
    N, D, K = 5001, 5, 1500
    T = rng.normal(size=(N, D))
    Y = T[rng.integers(0, N, K)] + 0.3 * rng.normal(size=(K, D))
    out = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DGTM_CTEMP_PAIRS", pairs)
        with pkg.Context(T, np.ones((K, 1)), "fp64") as c:
            c.set_Y(Y)
            c.estep(5.2, 1, 3.0)
            out.append(c.next_ctemp(1e9, 5.2, 1e-6, per_centre=True)[1])
    assert np.max(np.abs(out[0] / out[1] - 1.0)) <= 1e-13


@pytest.mark.parametrize("beta", [5e-324, 1e-310, 1e-200])
def test_vanishing_beta(pkg, beta):
    """beta so small that every exponent is 0 (its half too, for the smallest): R = 1 / K."""
    rng = np.random.default_rng(16)
    N, D, K = 900, 12, 64
    T, X = rng.normal(size=(N, D)), rng.normal(size=(K, 2))
    with pkg.Context(T, np.ones((K, 1)), "fp64") as c:
        assert c.path == "exact_slices"
        c.set_Y(rng.normal(size=(K, D)))
        c.estep(beta, 1, 1.5)
        R, M = c.R_block(0, K, 0, N), c.map(X)
    assert np.max(np.abs(R * K - 1.0)) <= 1e-15
    assert np.max(np.abs(M - X.mean(0))) <= 1e-14
