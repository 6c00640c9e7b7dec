"""The residual blocks' norms: one autograd node with the residual branch where nothing can tell, an ordinary call elsewhere."""
import pytest
import torch
from torch import nn

from fairscale_b200.models.gpt import Block, GPTConfig
from fairscale_b200.ops.norm import LayerNorm, RMSNorm, _NormResidualFn, norm_and_residual


def _block():
    torch.manual_seed(0)
    return Block(GPTConfig(vocab_size=32, d_model=16, n_heads=2, n_layers=1, ffn=32, max_seq=8))


def _fused(y):
    return y.grad_fn is not None and type(y.grad_fn).__name__ == _NormResidualFn.__name__ + "Backward"


def test_gradients_of_both_branches_add_up():
    x = torch.randn(2, 5, 16, requires_grad=True)
    for norm in (LayerNorm(16), RMSNorm(16)):
        h, r = norm_and_residual(norm, x)
        assert _fused(h)
        got = torch.autograd.grad((h * 3).sum() + (r * r).sum(), (x, *norm.parameters()))
        want = torch.autograd.grad((norm(x) * 3).sum() + (x * x).sum(), (x, *norm.parameters()))
        for a, b in zip(got, want):
            torch.testing.assert_close(a, b)


@pytest.mark.parametrize("make", [lambda: nn.LayerNorm(16), nn.Identity, lambda: nn.Sequential(LayerNorm(16))])
def test_any_module_may_stand_in_a_norms_place(make):
    block = _block()
    block.ln1, block.ln2 = make(), make()
    x = torch.randn(2, 8, 16, requires_grad=True)
    block(x).sum().backward()
    assert torch.isfinite(x.grad).all()


def test_hooks_see_the_norms_own_output():
    block = _block()
    seen = []
    block.ln1.register_forward_hook(lambda m, i, o: seen.append(o))
    block.ln2.register_forward_pre_hook(lambda m, i: seen.append(i[0]))
    x = torch.randn(2, 8, 16, requires_grad=True)
    plain = _block()(x)
    torch.testing.assert_close(block(x), plain)
    assert all(isinstance(t, torch.Tensor) and t.shape == x.shape for t in seen) and len(seen) == 2
    handle = nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(o) if isinstance(m, LayerNorm) else None)
    try:
        _block()(x)
    finally:
        handle.remove()
    assert len(seen) == 4 and all(isinstance(t, torch.Tensor) for t in seen)


def test_a_replaced_forward_is_run():
    norm = LayerNorm(16)
    norm.forward = lambda x: x * 2
    x = torch.randn(3, 16, requires_grad=True)
    h, r = norm_and_residual(norm, x)
    assert r is x and torch.equal(h, x * 2)


def test_a_stream_without_gradient_stays_without():
    norm, x = LayerNorm(16), torch.randn(3, 16)
    h, r = norm_and_residual(norm, x)
    assert r is x and not r.requires_grad and h.requires_grad
    r.add_(1.0)  # and may be changed in place
    with torch.no_grad():
        h, r = norm_and_residual(norm, x.requires_grad_())
    assert r is x and not h.requires_grad
