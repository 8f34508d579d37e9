"""poisson_nll's autograd function without a GPU: a stand-in for the model, whose likelihood and gradients are those of a
quadratic, in the layout that the kernels leave (params float32; background, Zernike and the value float64)."""
import numpy as np
import pytest
import torch

from insiliscope_b200.nll import poisson_nll


class Quadratic:
    """NLL = (|params|^2 + |bg|^2 + |zern|^2) / 2, so the gradients are the inputs."""

    def _eval(self, params, frame, bg, zern, counts, grad, want_mu=False):
        z = torch.as_tensor(zern).detach().to(torch.float64)
        p, b = params.detach().to(torch.float32), bg.detach().to(torch.float64)
        value = 0.5 * (p.double().square().sum() + b.square().sum() + z.square().sum())
        head = torch.stack([value, torch.zeros_like(value)])
        return float(value), head, None, ((p.clone(), b.clone(), z.clone()) if grad else None)

    def evaluate(self, params, frame, bg, zern, counts, grad=False, want_mu=False):
        value, _, mu, g = self._eval(params, frame, bg, zern, counts, grad, want_mu)
        return value, mu, g


def _inputs(zern_dtype=torch.float64):
    params = torch.tensor([[1.5, -2.0, 0.25, 3.0], [0.5, 4.0, -1.0, 2.0]], requires_grad=True)
    bg = torch.tensor([2.0, 0.125], requires_grad=True)
    return params, bg, torch.tensor([3, -1], dtype=zern_dtype)


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32, torch.float32, torch.float64])
def test_inputs_without_a_gradient_take_any_type(dtype):
    params, bg, zern = _inputs(dtype)
    poisson_nll(Quadratic(), params, bg, zern, None, None).backward()
    assert torch.equal(params.grad, params.detach()) and torch.equal(bg.grad, bg.detach())
    counts_bg = torch.tensor([2, 5], dtype=torch.int32)
    q = params.detach().clone().requires_grad_(True)
    poisson_nll(Quadratic(), q, counts_bg, zern, None, None).backward()
    assert torch.equal(q.grad, q.detach())


@pytest.mark.parametrize("zern", [np.array([3.0, -1.0]), [3.0, -1.0], torch.tensor([3.0, -1.0])])
def test_value_of_host_coefficients(zern):
    """Coefficients that are no tensor, where no gradient is wanted."""
    params, bg, _ = _inputs()
    want = 0.5 * sum(float(t.detach().double().square().sum()) for t in (params, bg)) + 5.0
    for p, b in ((params.detach(), bg.detach()), (params, bg)):
        with torch.no_grad():
            assert float(poisson_nll(Quadratic(), p, b, zern, None, None)) == want
    value = poisson_nll(Quadratic(), params.detach(), bg.detach(), zern, None, None)
    assert not value.requires_grad and value.dtype == torch.float64


def test_batched_gradients():
    """A batch of output gradients in one backward (what a vectorized Jacobian runs), and a differentiated backward."""
    params, bg, zern = _inputs()
    zern.requires_grad_(True)
    loss = poisson_nll(Quadratic(), params, bg, zern, None, None)
    go = torch.tensor([1.0, 0.3, -2.0], dtype=torch.float64)
    for grad, x in zip(torch.autograd.grad(loss, (params, bg, zern), go, is_grads_batched=True, retain_graph=True),
                       (params, bg, zern)):
        want = (go.reshape(-1, *[1] * x.dim()) * x.detach().double()).to(x.dtype)
        assert torch.equal(grad, want)
    s = torch.tensor(2.0, dtype=torch.float64, requires_grad=True)
    g, = torch.autograd.grad(s * loss, params, create_graph=True)
    d, = torch.autograd.grad(g.double().sum(), s)
    assert torch.equal(d, params.detach().double().sum())
