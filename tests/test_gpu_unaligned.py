"""Callers' FP32 arrays that start on 4 bytes only (a contiguous view at an odd element
offset): the same results, bit for bit, as from aligned copies, at even and odd D, on
the CUDA-core and the tensor-core paths."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def pair(N, K, D, seed=3):
    rng = np.random.default_rng(seed)
    T = rng.random((N, D)).astype(np.float32)
    Y = T[rng.integers(0, N, K)] + 0.05 * rng.standard_normal((K, D)).astype(np.float32)
    return torch.tensor(Y, device="cuda").contiguous(), torch.tensor(T, device="cuda").contiguous()


def shifted(x):
    """x in a buffer of its own, one float past an aligned start"""
    buf = torch.zeros(x.numel() + 1, dtype=x.dtype, device=x.device)
    v = buf[1:].view(x.shape)
    v.copy_(x)
    assert v.is_contiguous() and v.data_ptr() % 8 == 4
    return v


@pytest.mark.parametrize("D", [2, 12, 33, 64, 166, 190, 200, 255, 256])
@pytest.mark.parametrize("which", ["Y", "T", "both"])
def test_free_energy_on_unaligned_tensors(pkg, D, which):
    ag = importlib.import_module(pkg.__name__ + ".autograd")
    out = []
    for odd in (False, True):
        Y, T = pair(700, 130, D)
        if odd and which in ("Y", "both"):
            Y = shifted(Y)
        if odd and which in ("T", "both"):
            T = shifted(T)
        beta = torch.tensor(8.0, dtype=torch.float64, device="cuda", requires_grad=True)
        F = ag.free_energy(Y.requires_grad_(True), T.requires_grad_(True), beta, 1.3)
        out.append([F.detach()] + list(torch.autograd.grad(F, (Y, T, beta))))
        torch.cuda.synchronize()
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("D", [2, 12, 33, 64, 100, 166, 200, 256])
def test_forward_noalloc_on_unaligned_tensors(pkg, D):
    lib = pkg.load_library()
    stream = torch.cuda.current_stream().cuda_stream
    Y, T = pair(700, 130, D)
    out = []
    for a, b in ((Y, T), (shifted(Y), T), (Y, shifted(T)), (shifted(Y), shifted(T))):
        F = torch.empty((), dtype=torch.float64, device="cuda")
        rc = lib.dgtm_fe_forward_noalloc(ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), 700, 130, D,
                                         ctypes.c_double(8.0), ctypes.c_double(1.3), ctypes.c_void_p(stream),
                                         ctypes.c_void_p(F.data_ptr()))
        assert rc == 0, lib.dgtm_last_error_string()
        torch.cuda.synchronize()
        out.append(F.item())
    assert len(set(out)) == 1
