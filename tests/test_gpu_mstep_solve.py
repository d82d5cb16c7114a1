"""The M-step's solve at the sizes where its kernels change: W against a host
FP64 solve of the same normal equations, formed from the context's own G and
RT.  Two backward-stable solvers of A W = B differ by a modest multiple of
M1 eps cond(A); the bound is 8 M1 eps cond(A), in Frobenius norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve_case(pkg, M1, D, K, solver, precision="fp64"):
    rng = np.random.default_rng(1000 * M1 + D)
    T = rng.random((260, D))
    FI = np.concatenate([rng.random((K, M1 - 1)), np.ones((K, 1))], axis=1)
    with pkg.Context(T, FI, precision, solver=solver) as c:
        c.set_Y(rng.random((K, D)))
        c.estep(2.0, 1, 1.5)
        _, W, _ = c.mstep()
        G, RT = c.get_stats()
    A, B = FI.T @ (G[:, None] * FI), FI.T @ RT
    ref = np.linalg.solve(A, B)
    tol = 8 * M1 * np.finfo(float).eps * np.linalg.cond(A)
    assert np.linalg.norm(W - ref) <= tol * np.linalg.norm(ref)


# odd and even orders, one pair, the last size in shared memory and the first beyond it
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("M1,D", [(1, 3), (2, 5), (3, 1), (26, 9), (65, 33), (112, 6), (113, 6)])
def test_svd_sizes(pkg, M1, D, precision):
    solve_case(pkg, M1, D, 3 * M1 + 20, "svd", precision)


# the normal equations by digit slices: one tile and several, ragged K, M1 and D,
# contractions of one segment (512 centres) and of many
@pytest.mark.parametrize("K,M1,D", [(8000, 65, 166), (5003, 129, 33), (1500, 513, 7), (2111, 200, 190),
                                    (33000, 30, 64), (700, 250, 20)])
def test_normal_equations_by_slices(pkg, K, M1, D):
    solve_case(pkg, M1, D, K, "cholesky")


# the blocked Cholesky and the two substitutions: the last order in shared memory, the
# first beyond it, whole and partial panels, every register bucket; the multiply-add
# normal equations of the FP32 form at tiles of 64 that are only partly filled
@pytest.mark.parametrize("M1,D,precision", [(32, 3, "fp64"), (33, 65, "fp32"), (110, 7, "fp32"), (111, 7, "fp32"),
                                            (128, 64, "fp32"), (129, 2, "fp32"), (257, 5, "fp32"),
                                            (400, 6, "fp64"), (513, 9, "fp32"), (700, 3, "fp64")])
def test_cholesky_sizes(pkg, M1, D, precision):
    solve_case(pkg, M1, D, 2 * M1 + 20, "cholesky", precision)
