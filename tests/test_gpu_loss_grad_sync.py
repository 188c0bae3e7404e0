"""The objective and gradient call is synchronous: when it returns, the gradient is complete,
so that another stream may read it.  At 512^3 the last pass takes some hundred microseconds,
longer than the return takes: a call that did not wait leaves the stream busy."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lam", [0.0, 1e-3])
def test_gradient_is_complete(dev, lam):
    import torch
    import ctdm_gb300 as C
    r = 512
    F2 = torch.zeros((r, r, r), dtype=torch.complex64, device=dev)
    F2[::7, ::3, ::2] = 1 + 1j
    tape = C.Tape(F2, r, 4.0)
    V = torch.full((r, r, r), 0.1 + 0.1j, dtype=torch.complex64, device=dev)
    g = torch.zeros_like(V)
    for _ in range(3):
        torch.cuda.synchronize()
        tape.loss_grad(V, g, lam)
        assert torch.cuda.default_stream(dev).query()
    tape.close()
