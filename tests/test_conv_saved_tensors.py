"""The convolution's backward pass on tensors that are not as its forward pass made
them: saved tensors that hooks return elsewhere or in another layout, and output
gradients that are not contiguous.  The same values as without hooks."""
import pytest

pytestmark = pytest.mark.gpu

SHAPE, CIN, COUT = (2, 9, 21), 16, 32


def _grads(unpack=None, dy=None):
    import torch
    from skewengine_gb300 import surrogate as sur
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((*SHAPE, CIN), generator=g, device="cuda").to(torch.bfloat16).requires_grad_(True)
    w = torch.randn((COUT, sur.kpad(CIN)), generator=g, device="cuda").requires_grad_(True)
    b = torch.randn(COUT, generator=g, device="cuda").requires_grad_(True)
    if dy is None:
        dy = torch.randn((*SHAPE, COUT), generator=g, device="cuda").to(torch.bfloat16)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack or (lambda t: t)):
        y = sur.conv_op(x, w, b, True)
        return torch.autograd.grad(y, (x, w, b), dy)


def _agree(got, want):
    import torch
    assert torch.equal(got[0], want[0])
    assert torch.allclose(got[1], want[1], rtol=1e-5, atol=1e-5)  # atomics in any order
    assert torch.allclose(got[2], want[2], rtol=1e-6, atol=1e-6)


def _moved(t, by):
    """t, starting `by` elements past an allocation."""
    import torch
    flat = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    out = flat[by:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("what", ["output off its alignment", "output in another layout", "weights in another layout"])
def test_hooks_that_return_other_layouts(gpu_lib, what):
    def unpack(t):
        if what == "output off its alignment" and t.shape[-1] == COUT and t.dim() == 4:
            return _moved(t, 1)
        if what == "output in another layout" and t.shape[-1] == COUT and t.dim() == 4:
            return t.permute(3, 0, 1, 2).contiguous().permute(1, 2, 3, 0)
        if what == "weights in another layout" and t.dim() == 2:
            return t.t().contiguous().t()
        return t
    _agree(_grads(unpack), _grads())


@pytest.mark.parametrize("kind", ["expanded", "permuted"])
def test_output_gradients_that_are_not_contiguous(gpu_lib, kind):
    import torch
    if kind == "expanded":
        dy = torch.full((), 0.5, dtype=torch.bfloat16, device="cuda").expand(*SHAPE, COUT)
    else:
        dy = torch.randn((COUT, *SHAPE), device="cuda").to(torch.bfloat16).permute(1, 2, 3, 0)
    _agree(_grads(dy=dy), _grads(dy=dy.contiguous()))
