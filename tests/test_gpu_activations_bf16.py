"""bf16 activations (forward and gradient) over every bf16 number against fp64, and at the edges of the kernels' batches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _every():
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    return x[torch.isfinite(x)]


def _exact(x, name):
    x = x.double()
    if name == "relu":
        return x.clamp(min=0), (x > 0).double()
    if name == "gelu":
        k0, k1 = (2 / torch.pi) ** 0.5, 0.044715
        s = torch.sigmoid(2 * k0 * (x + k1 * x ** 3))
        return x * s, s + x * s * torch.sigmoid(-2 * k0 * (x + k1 * x ** 3)) * 2 * k0 * (1 + 3 * k1 * x * x)
    s = torch.sigmoid(x)
    if name == "sigmoid":
        return s, s * torch.sigmoid(-x)
    if name == "tanh":
        return torch.tanh(x), 1 / torch.cosh(x) ** 2
    return x * s, s + x * s * torch.sigmoid(-x)


@pytest.mark.parametrize("name", ["relu", "gelu", "sigmoid", "tanh", "silu"])
def test_every_number(name):
    from ghost_flow_b200 import ops

    x = _every()
    x = x[x.abs() < 60].clone()               # beyond that the function is its limit and x^3 leaves fp32 in the gradient
    x = x[:x.numel() // 8 * 8].requires_grad_()
    y = ops.unary(x, name)
    y.backward(torch.ones_like(y))
    want, grad = _exact(x.detach(), name)
    # eight bits of the result: 2^-8 at most, computed in fp32 with exponentials of arguments up to 150: 2^-24 x 150 of them. A
    # gradient is a sum of terms of size one, and so is what is lost there: 2^-20. Numbers below 2^-126 are flushed.
    assert ((y.double() - want).abs() <= 2 ** -7.99 * want.abs() + 2 ** -20 * (name != "relu")).all()
    assert ((x.grad.double() - grad).abs() <= 2 ** -7.99 * grad.abs() + 2 ** -18).all()
    if name == "gelu":                        # small results keep their digits: x sigmoid(2 u), not x (1 + tanh u) / 2
        m = (want.abs() > 1e-30) & (x.detach().double() < -3)
        assert ((y.double() - want).abs() <= 2 ** -7.99 * want.abs())[m].all()


@pytest.mark.parametrize("n", [8, 2048, 8192, 8200, 16384 + 8, 1 << 20])
def test_batches(n):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, generator=g, device="cuda").bfloat16().requires_grad_()
    dy = torch.randn(n, generator=g, device="cuda").bfloat16()
    y = ops.gelu(x)
    y.backward(dy)
    want, grad = _exact(x.detach(), "gelu")
    assert torch.allclose(y.double(), want, rtol=2 ** -8, atol=2 ** -20)
    assert torch.allclose(x.grad.double(), grad * dy.double(), rtol=2 ** -8, atol=2 ** -17)


@pytest.mark.parametrize("T,F", [(1, 8), (3, 520), (1, 4096), (511, 24), (129, 1376), (2, 8200)])
def test_swiglu(T, F):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + F)
    gu = torch.randn(T, 2 * F, generator=g, device="cuda").bfloat16().requires_grad_()
    dy = torch.randn(T, F, generator=g, device="cuda").bfloat16()
    y = ops.swiglu(gu)
    y.backward(dy)
    r = gu.detach().double().requires_grad_()
    a, b = r.chunk(2, -1)
    want = torch.nn.functional.silu(a) * b
    (grad,) = torch.autograd.grad(want, r, dy.double())
    assert torch.allclose(y.double(), want, rtol=2 ** -8, atol=2 ** -20)
    assert torch.allclose(gu.grad.double(), grad, rtol=2 ** -8, atol=2 ** -17)


@pytest.mark.parametrize("name", ["gelu", "silu", "relu"])
def test_infinities_and_nan(name):
    from ghost_flow_b200 import ops

    x = torch.tensor([float("inf"), float("nan"), 0.0, 3e38, -3e38, 1.0, -1.0, 2.0], device="cuda").bfloat16()
    y = ops.unary(x, name)
    assert y[0] == float("inf") and (torch.isnan(y[1]) or name == "relu") and y[2] == 0 and y[3] == x[3] and y[4] == 0


@pytest.mark.parametrize("name", ["relu", "gelu", "sigmoid", "tanh", "silu"])
def test_numbers_of_any_size(name):
    """Beyond what ``test_every_number`` takes, up to the largest finite number, where squares and cubes leave fp32."""
    from ghost_flow_b200 import ops

    x = _every()
    x = x[x.abs() >= 60]
    x = torch.cat((x, x[:-x.numel() % 8])).requires_grad_()
    y = ops.unary(x, name)
    y.backward(torch.ones_like(y))
    want, grad = _exact(x.detach(), name)          # 3e38 squared and cubed are finite in fp64
    assert ((y.double() - want).abs() <= 2 ** -7.99 * want.abs() + 2 ** -20 * (name != "relu")).all()
    assert ((x.grad.double() - grad).abs() <= 2 ** -7.99 * grad.abs() + 2 ** -18).all()


@pytest.mark.parametrize("n", [(8 << 20) - 8, 8 << 20, (8 << 20) + 8, (20 << 20) - 8, (20 << 20) + 2056])
@pytest.mark.parametrize("name", ["gelu", "silu"])
def test_numbers_of_vectors_to_a_thread(n, name):
    """Around the sizes where a thread gets more vectors."""
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, generator=g, device="cuda").bfloat16().requires_grad_()
    dy = torch.randn(n, generator=g, device="cuda").bfloat16()
    y = ops.unary(x, name)
    y.backward(dy)
    want, grad = _exact(x.detach(), name)
    assert torch.allclose(y.double(), want, rtol=2 ** -8, atol=2 ** -20)
    assert torch.allclose(x.grad.double(), grad * dy.double(), rtol=2 ** -8, atol=2 ** -17)


@pytest.mark.parametrize("T,F", [(6143, 1024), (6144, 1024), (6145, 1024), (4095, 8192), (4096, 8192), (700, 11008)])
def test_swiglu_numbers_of_vectors(T, F):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + F)
    gu = torch.randn(T, 2 * F, generator=g, device="cuda").bfloat16().requires_grad_()
    dy = torch.randn(T, F, generator=g, device="cuda").bfloat16()
    y = ops.swiglu(gu)
    y.backward(dy)
    a, b = gu.detach().double().chunk(2, -1)
    s = torch.sigmoid(a)
    assert torch.allclose(y.double(), a * s * b, rtol=2 ** -8, atol=2 ** -20)
    want = torch.cat((dy.double() * b * (s + a * s * (1 - s)), dy.double() * a * s), -1)
    assert torch.allclose(gu.grad.double(), want, rtol=2 ** -8, atol=2 ** -17)
