"""The graph node of the differentiable entry under the other mechanisms of autograd."""

import pytest
import torch

pytestmark = pytest.mark.gpu

Z, H, HK, S, D = 1, 4, 2, 200, 128


def _inputs(dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(3)
    return [torch.randn(Z, n, S, D, device="cuda", dtype=dtype, generator=g) for n in (H, HK, HK, H)]


def _attend(q, k, v, **kw):
    import sageattention_b200.nvfp4 as nv
    return nv.nvfp4_flash_attn_func(q, k, v, D ** -0.5, causal=True, num_key_value_groups=H // HK, **kw)


@pytest.mark.parametrize("which", [0, 1, 2, 3])
@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_is_refused(which, grad):
    """A tangent on any operand raises (as an autograd.Function without a jvp does); it is not dropped."""
    import torch.autograd.forward_ad as fw
    q, k, v, _ = _inputs(torch.float32)
    bias = torch.zeros(Z, S, device="cuda")
    ops = [q, k, v, bias]
    ops[0].requires_grad_(grad)
    with fw.dual_level():
        ops[which] = fw.make_dual(ops[which], torch.ones_like(ops[which]))
        with pytest.raises(NotImplementedError, match="forward"):
            _attend(*ops[:3], key_pad_bias=ops[3])
    assert _attend(q, k, v, key_pad_bias=bias).shape == (Z, H, S, D)


def test_function_transforms_are_refused():
    q, k, v, _ = _inputs()
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda q: _attend(q, k, v).float().sum())(q)
    with pytest.raises(RuntimeError):
        torch.func.vmap(_attend)(q[None], k[None], v[None])
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.jvp(lambda q: _attend(q, k, v), (q,), (q,))


@pytest.mark.parametrize("operands", [False, True])
def test_bias_that_requires_a_gradient(operands):
    """The bias gets no gradient; the output is part of the graph all the same, and backward runs."""
    q, k, v, do = _inputs()
    for t in (q, k, v):
        t.requires_grad_(operands)
    bias = torch.zeros(Z, S, device="cuda", requires_grad=True)
    out = _attend(q, k, v, key_pad_bias=bias)
    assert out.requires_grad
    out.backward(do)
    assert bias.grad is None and all((t.grad is not None) == operands for t in (q, k, v))
