"""Failure detection without a GPU fault: every wait in the tensor-core
kernels is bounded by a wall-clock limit, records a site code when it gives
up, and the host reports DGTM_ETIMEOUT.  Here one such wait runs out on a
barrier that nothing arrives at (50 ms limit); the error reaches the host
and the device keeps working."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_bounded_wait_gives_up_and_device_stays_usable(pkg, orc):
    code, site, ms = pkg.wait_probe(50)
    assert code == 5  # DGTM_ETIMEOUT
    assert site == 90
    assert 50.0 <= ms < 2000.0
    msg = pkg.load_library().dgtm_last_error_string().decode()
    assert "gave up" in msg and "site 90" in msg
    # the tensor-core kernels and a whole EM step still run afterwards
    assert pkg.selftest() == [0.0, 0.0, 0.0, 0.0]
    ds = importlib.import_module(pkg.__name__ + ".datasets")
    st = importlib.import_module(pkg.__name__ + ".gtm_setup")
    T = ds.fingerprints(600, 40, 8, seed=4)
    X, FI = st.setup_grid(2, 64, 9, 1.0)
    rng = np.random.default_rng(4)
    Y = T[rng.integers(0, 600, 64)] * 0.7 + 0.15
    R, vgc, vgc2 = orc.resp(orc.dist(Y, T), 1.0, 1, 2.0)
    with pkg.Context(T, FI, "bf16x3") as c:
        c.set_Y(Y)
        llh, nfree = c.estep(1.0, 1, 2.0)
        c.mstep()
    assert llh == pytest.approx(orc.qual(600, 64, 40, 1.0, vgc, 0, 2.0), rel=1e-5)


def test_wait_probe_rejects_bad_limits(pkg):
    code, _, _ = pkg.wait_probe(0)
    assert code == 1  # DGTM_EINVAL


def test_gradients_are_nan_once_a_wait_gave_up(pkg):
    """A wait of the free energy's passes that gave up (here its record, written into the
    workspace by hand) makes every gradient NaN as a whole; cleared, the same workspace
    gives the gradients again."""
    import ctypes
    torch = pytest.importorskip("torch")
    lib = pkg.load_library()
    N, K, D = 3001, 300, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    T = torch.rand((N, D), device="cuda", generator=g)
    Y = torch.rand((K, D), device="cuda", generator=g)
    size = ctypes.c_size_t()
    assert lib.dgtm_fe_workspace_size(N, K, D, ctypes.byref(size)) == 0
    ws = torch.zeros(size.value + 256, dtype=torch.uint8, device="cuda")
    at = -ws.data_ptr() % 256
    ptr, stream = ws.data_ptr() + at, torch.cuda.current_stream().cuda_stream
    F, one, db = (torch.ones((), dtype=torch.float64, device="cuda") for _ in range(3))

    def backward():
        dY, dT = torch.zeros_like(Y), torch.zeros_like(T)
        assert lib.dgtm_fe_backward(Y.data_ptr(), T.data_ptr(), N, K, D, 5.0, 1.2, ptr, size.value, stream,
                                    one.data_ptr(), dY.data_ptr(), dT.data_ptr(), db.data_ptr()) == 0
        torch.cuda.synchronize()
        return dY, dT, db.clone()

    assert lib.dgtm_fe_forward(Y.data_ptr(), T.data_ptr(), N, K, D, 5.0, 1.2, ptr, size.value, stream,
                               F.data_ptr()) == 0
    good = backward()
    assert all(bool(torch.isfinite(x).all()) for x in good)
    word = ws[at + size.value - 256:at + size.value - 252].view(torch.int32)  # the workspace's last slot
    word.fill_(41)
    bad = backward()
    assert all(bool(torch.isnan(x).all()) for x in bad)
    word.fill_(0)
    for a, b in zip(good, backward()):
        assert torch.equal(a, b)
