"""The digit-slice E-step, responsibility pass and map (real-valued data of the
FP64 form, and the map of every form) against the oracle, at the sizes where
tiles, panels and chunks are only partly filled.  The FP64 form's stated bounds
apply: 1e-12 relative on the qualities, G, RT and the map, 1e-13 on R."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def problem(N, D, K, seed, scale=None, binary=False):
    rng = np.random.default_rng(seed)
    T = (rng.random((N, D)) < 0.4).astype(float) if binary else rng.normal(size=(N, D))
    Y = rng.normal(size=(K, D)) * 0.7
    if scale is not None:
        s = np.logspace(-scale, scale, D)
        T, Y = T * s, Y * s
    FI = np.concatenate([rng.random((K, 3)), np.ones((K, 1))], axis=1)
    return T, Y, FI, rng.normal(size=(K, 3))


def oracle(orc, T, Y, beta, isDA, temp):
    R, vgc, vgc2 = orc.resp(orc.dist(Y, T), beta, isDA, temp)
    N, D = T.shape
    K = Y.shape[0]
    llh = orc.qual(N, K, D, beta, vgc, 0, temp)
    return R, llh, orc.qual(N, K, D, beta, vgc2, 1, temp) if isDA else -llh


# one panel and four, one dimension, ragged N and K, one chunk and several
# (chunks hold 8 M pairs, 128 points at least), both temperatures, plain EM
@pytest.mark.parametrize("N,D,K,isDA,temp,scale", [
    (256, 1, 8000, 1, 1.5, None), (4001, 3, 517, 1, 1.0, None), (2050, 64, 1001, 1, 2.0, None),
    (2177, 65, 8000, 1, 1.3, None), (1000, 130, 2049, 0, 1.0, None), (700, 200, 3000, 1, 3.0, None),
    (513, 256, 4097, 1, 2.0, None), (3000, 12, 700, 1, 1.2, 2.0), (90001, 7, 130, 1, 2.0, None)])
def test_em_step_and_map(pkg, orc, N, D, K, isDA, temp, scale):
    T, Y, FI, X = problem(N, D, K, N + D, scale)
    beta = 2.0 / max(1.0, np.mean(np.sum(T * T, axis=1)) / 8)
    with pkg.Context(T, FI, "fp64") as c:
        assert c.path == "exact_slices"
        c.set_Y(Y)
        llh, nfree = c.estep(beta, isDA, temp)
        M = c.map(X)
        Rb = c.R_block(0, 17, 0, N)
        c.mstep()
        G, RT = c.get_stats()
    R, ollh, onfree = oracle(orc, T, Y, beta, isDA, temp)
    assert llh == pytest.approx(ollh, rel=1e-12)
    assert nfree == pytest.approx(onfree, rel=1e-12)
    assert np.max(np.abs(Rb - R[:17])) <= 1e-13
    assert rel(G, R.sum(1)) <= 1e-12
    assert rel(RT, R @ T) <= 1e-12
    assert rel(M, R.T @ X) <= 1e-12


def test_far_centre_keeps_its_statistics(pkg, orc):
    """A centre whose largest responsibility is far below 2^-56 keeps G and RT to
    the form's relative accuracy (its own power-of-two grid)."""
    T, Y, FI, X = problem(3000, 5, 700, 1)
    Y[3] = 8.0
    beta, temp = 1.0, 1.1
    R, _, _ = oracle(orc, T, Y, beta, 1, temp)
    assert 0 < R[3].max() < 1e-20
    with pkg.Context(T, FI, "fp64") as c:
        c.set_Y(Y)
        c.estep(beta, 1, temp)
        c.mstep()
        G, RT = c.get_stats()
    assert G[3] == pytest.approx(R[3].sum(), rel=1e-10)
    assert rel(RT[3], R[3] @ T) <= 1e-10


def test_zero_column_and_nonfinite_centre(pkg, orc):
    T, Y, FI, X = problem(3000, 4, 700, 2)
    T[5] = 500.0  # exp(-beta d / 2) underflows for every centre
    with pkg.Context(T, FI, "fp64") as c:
        c.set_Y(Y)
        llh, nfree = c.estep(4.0, 1, 1.5)
        assert llh == -np.inf and np.isfinite(nfree)
        assert np.max(np.abs(c.R_block(0, 20, 5, 1) - 1 / 700)) <= 1e-15
        M = c.map(X)
        assert np.max(np.abs(M[5] - X.mean(0))) <= 1e-12
        Y[7, 2] = np.nan
        c.set_Y(Y)
        llh, nfree = c.estep(4.0, 1, 1.5)
        assert np.isnan(llh) and np.isnan(nfree)


@pytest.mark.parametrize("form,binary,D", [("bf16x3", True, 166), ("bf16x3", False, 64), ("fp32", False, 31),
                                           ("fp64", True, 100), ("fp32", True, 200)])
def test_map_matches_cuda_cores(pkg, monkeypatch, form, binary, D):
    """The map of every form against the CUDA-core map kernel on the same column
    statistics."""
    T, Y, FI, X = problem(2100, D, 1050, D, binary=binary)
    Y = 0.4 + 0.2 * Y if binary else Y
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("DGTM_X64", on if form != "fp64" else "1")
        with pkg.Context(T, FI, form) as c:
            c.set_Y(Y)
            c.estep(1.5, 1, 1.2)
            monkeypatch.setenv("DGTM_X64", on)
            out.append(c.map(X))
    assert rel(out[0], out[1]) <= 1e-12


# few depths, whose products are 64-bit integers: both sides of every row length and of
# the switch to digits, points and centres off the blocks of 256 and 64
@pytest.mark.parametrize("N,D,K", [(520, 1, 65), (300, 2, 129), (257, 3, 130), (1030, 4, 64), (511, 5, 67),
                                   (700, 8, 81), (513, 9, 66)])
def test_few_depths(pkg, N, D, K):
    """Responsibilities against extended precision.  Their relative error is c times
    the errors of the distances to the centre and to the nearest one, two roundings
    of |y|^2 / 2 and an integer unit each (under 2^-51 |y|^2 + 2^-53 |t||y| D), and a few
    roundings of the exponent, its sum's logarithm and the result."""
    T, Y, FI, X = problem(N, D, K, N + D)
    beta, temp = 6.0, 1.5
    with pkg.Context(T, FI, "fp64") as c:
        assert c.path == "exact_slices"
        c.set_Y(Y)
        c.estep(beta, 1, temp)
        R = c.R_block(0, K, 0, N)
    q = np.longdouble
    d = ((T[None].astype(q) - Y[:, None].astype(q)) ** 2).sum(2)
    v = -d * (q(beta) / 2 / q(temp))
    e = np.exp(v - v.max(0))
    ref = e / e.sum(0)
    y2, t2 = np.max(np.sum(Y * Y, 1)), np.max(np.sum(T * T, 1))
    arg = float(-(v - v.max(0)).min()) + np.log(K)
    tol = beta / (2 * temp) * 2 * (2.0**-51 * y2 + 2.0**-53 * D * np.sqrt(y2 * t2)) + 2.0**-52 * (arg + 4)
    assert np.max(np.abs(R - ref) / ref) <= tol


# the FP64 critical temperatures by digit slices against the CUDA-core scatter,
# centre by centre: two dimensions, one and several tiles of features and of
# centres, several batches of centres (a small budget), several chunks of points
@pytest.mark.parametrize("N,D,K,binary,mb", [
    (7000, 2, 4001, False, 8192), (2000, 65, 1001, False, 8192), (2100, 20, 1500, False, 64),
    (9000, 33, 1301, False, 8192), (2500, 40, 900, True, 8192), (20000, 64, 125, False, 8192)])
def test_ctemp_matches_cuda_cores(pkg, monkeypatch, N, D, K, binary, mb):
    T, Y, FI, _ = problem(N, D, K, N + D, binary=binary)
    beta = 8.0 / D
    out = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DGTM_CTEMP_PAIRS", pairs)
        monkeypatch.setenv("DGTM_CTEMP_GEMM_MB", str(mb))
        with pkg.Context(T, FI, "fp64") as c:
            c.set_Y(Y if not binary else 0.4 + 0.2 * Y)
            c.estep(beta, 1, 2.0)
            out.append(c.next_ctemp(50.0, beta, 1e-6, per_centre=True))
    (a, ak), (b, bk) = out
    assert a == pytest.approx(b, rel=1e-12)
    # the expansion may cancel 8 bits of 2^-53: 2.8e-14 of the largest eigenvalue
    assert np.max(np.abs(ak - bk) / bk) <= 1e-13


def test_ctemp_tight_clusters_are_redone(pkg, monkeypatch):
    """Clusters of width 1e-4 far from the mean: the expansion would cancel 24
    bits, so those centres go through the CUDA-core scatter."""
    rng = np.random.default_rng(3)
    mu = rng.normal(size=(700, 8))
    T = mu[rng.integers(0, 700, 4000)] + 1e-4 * rng.normal(size=(4000, 8))
    FI = np.ones((700, 1))
    out = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DGTM_CTEMP_PAIRS", pairs)
        with pkg.Context(T, FI, "fp64") as c:
            c.set_Y(mu)
            c.estep(1e5, 1, 1.5)
            out.append(c.next_ctemp(1e6, 1e5, 1e-6, per_centre=True)[1])
    np.testing.assert_allclose(out[0], out[1], rtol=1e-13)  # zeros and HUGE_VAL alike


@pytest.mark.parametrize("N,D,K,k0,nk,n0,nn", [(5000, 20, 3000, 2900, 100, 4871, 129),
                                               (5000, 20, 3000, 1, 3, 127, 4000), (70000, 3, 500, 63, 130, 1, 69999),
                                               (300, 5, 200, 199, 1, 299, 1)])
def test_r_blocks(pkg, orc, N, D, K, k0, nk, n0, nn):
    """Blocks that start and end off the tiles, from kept distances and from
    recomputed ones, and the M-step after them."""
    T, Y, FI, X = problem(N, D, K, K + nk)
    beta, temp = 2.0, 1.4
    with pkg.Context(T, FI, "fp64") as c:
        c.set_Y(Y)
        c.estep(beta, 1, temp)
        Rb = c.R_block(k0, nk, n0, nn)
        c.mstep()
        G, _ = c.get_stats()
    R, _, _ = oracle(orc, T, Y, beta, 1, temp)
    assert np.max(np.abs(Rb - R[k0:k0 + nk, n0:n0 + nn])) <= 1e-13
    assert rel(G, R.sum(1)) <= 1e-12
