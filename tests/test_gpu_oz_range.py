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
    normal = R[9] > 1e-300
    # an exponent of 600 nats carries 600 x 2^-53 x a few
    assert np.max(np.abs(Rb[normal] / R[9][normal] - 1.0)) <= 1e-11
    gk = R[9].sum()
    assert G[9] == pytest.approx(gk, rel=1e-11)
    assert np.max(np.abs(RT[9] - R[9] @ T)) <= 1e-11 * np.max(np.abs(R[9] @ T))
    assert np.isfinite(got_k[9]) and np.isfinite(got) and got == np.max(got_k)
