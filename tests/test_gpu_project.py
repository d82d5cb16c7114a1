"""Arguments of the projection: step sizes as tensors, and what it refuses."""
import importlib

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture
def case(pkg):
    g = torch.Generator(device="cuda").manual_seed(2)
    T = torch.rand((501, 20), device="cuda", generator=g)
    Y = torch.rand((90, 20), device="cuda", generator=g)
    return importlib.import_module(pkg.__name__ + ".autograd"), T, Y


def test_step_size_as_a_tensor(case):
    ag, T, Y = case
    ref = ag.project(T, Y, 5.0, 1.2, steps=4, lr=0.125)
    # g * 2^-3 is exact, so the number's fused multiply-add rounds alike
    for lr in (torch.tensor(0.125, device="cuda"), torch.full((501, 1), 0.125, device="cuda"),
               torch.full((20,), 0.125, device="cuda"), torch.tensor(0.125, device="cuda", requires_grad=True)):
        got = ag.project(T, Y, 5.0, 1.2, steps=4, lr=lr)
        assert torch.equal(got, ref) and not got.requires_grad
    lr = torch.zeros((501, 1), device="cuda")
    lr[7] = 0.125
    got = ag.project(T, Y, 5.0, 1.2, steps=4, lr=lr)
    assert torch.equal(got[7], ref[7]) and torch.equal(got[:7], T[:7]) and torch.equal(got[8:], T[8:])


def test_refusals(case):
    ag, T, Y = case
    with pytest.raises(RuntimeError):
        ag.project(T.int(), Y, 5.0, steps=0)
    with pytest.raises(TypeError):
        ag.project(T, Y, 5.0, steps=0.5)
    with pytest.raises(TypeError):
        ag.project(T.double(), Y, 5.0)
    with torch.no_grad():
        with pytest.raises(RuntimeError):
            ag.project(T, Y, 5.0)
        with pytest.raises(TypeError):
            ag.project(T.double(), Y, 5.0)
    assert torch.equal(ag.project(T, Y, 5.0, steps=0), T)
