"""The FP32 form's two passes at the edges of their tiles (64 points, 64 and 32
centres, rows of 4 and 32 depths) against the oracle: the form's stated 1e-5 on
the qualities and 1e-4 on G and RT."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,D,K,isDA", [(1, 1, 1, 1), (63, 4, 31, 1), (65, 5, 33, 1), (64, 31, 64, 0),
                                        (200, 33, 65, 1), (1000, 166, 129, 1), (321, 224, 70, 1),
                                        (130, 256, 100, 1)])
def test_tiles(pkg, orc, N, D, K, isDA):
    rng = np.random.default_rng(N + D + K)
    T, Y = rng.random((N, D)), rng.random((K, D))
    FI = np.concatenate([rng.random((K, 2)), np.ones((K, 1))], axis=1)
    beta, temp = 3.0, 1.4 if isDA else 1.0
    R, vgc, vgc2 = orc.resp(orc.dist(Y, T), beta, isDA, temp)
    ollh = orc.qual(N, K, D, beta, vgc, 0, temp)
    onfree = orc.qual(N, K, D, beta, vgc2, 1, temp) if isDA else -ollh
    with pkg.Context(T, FI, "fp32") as c:
        c.set_Y(Y)
        llh, nfree = c.estep(beta, isDA, temp)
        try:
            c.mstep()
        except pkg.DgtmError as e:  # a degenerate exact fit gives beta = inf
            assert e.code == 4
        G, RT = c.get_stats()
    assert llh == pytest.approx(ollh, rel=1e-5)
    assert nfree == pytest.approx(onfree, rel=1e-5)
    assert np.max(np.abs(G - R.sum(1))) <= 1e-4 * np.max(R.sum(1))
    assert np.max(np.abs(RT - R @ T)) <= 1e-4 * np.max(np.abs(R @ T))


def test_zero_column(pkg):
    rng = np.random.default_rng(5)
    T, Y = rng.random((100, 6)), rng.random((40, 6))
    T[7] = 300.0
    with pkg.Context(T, np.ones((40, 1)), "fp32") as c:
        c.set_Y(Y)
        llh, nfree = c.estep(5.0, 1, 1.5)
        assert llh == -np.inf and np.isfinite(nfree)
        c.mstep()
        G, _ = c.get_stats()
    assert abs(G.sum() - 100) <= 1e-4
