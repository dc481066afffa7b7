"""The ReLU and bias gradient where a thread takes several pixels and the blocks are
all in use (608 blocks of 256 / (C / 8) pixels), with remainders; and the whole
backward call at such a size, with and without the ReLU and the data gradient."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 131, 129, 64), (1, 37, 41, 2048), (2, 300, 301, 8)]


def _inputs(shape):
    import torch
    g = torch.Generator(device="cuda").manual_seed(shape[2])
    dy = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    y = torch.randn(shape, generator=g, device="cuda").clamp_min_(0).to(torch.bfloat16)
    return dy, y


def _sums_agree(db, dz):
    """Plain additions of a thread's pixels, at most 32 here, everything after with
    the roundings carried along and one at the end."""
    ref, mag = dz.double().sum((0, 1, 2)), dz.double().abs().sum((0, 1, 2))
    assert bool(((db.double() - ref).abs() <= 34 * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_relu_grad_with_several_pixels_a_thread(gpu_lib, shape, relu):
    import torch
    from skewengine_gb300 import surrogate as sur
    assert shape[0] * shape[1] * shape[2] > 608 * 256 // (shape[3] // 8)
    dy, y = _inputs(shape)
    dz, db = sur.relu_grad(dy, y if relu else None)
    want = dy * (y > 0) if relu else dy
    assert torch.equal(dz.view(torch.int16), want.view(torch.int16))
    _sums_agree(db, want)


@pytest.mark.parametrize("need_dx", [False, True])
@pytest.mark.parametrize("relu", [False, True])
def test_backward_with_several_pixels_a_thread(gpu_lib, relu, need_dx):
    import torch
    from skewengine_gb300 import surrogate as sur
    n, h, w, cout, cin = 3, 131, 129, 64, 32
    dy, y = _inputs((n, h, w, cout))
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((n, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    wt = torch.randn((cout, sur.kpad(cin)), generator=g, device="cuda").to(torch.bfloat16)
    dx, dw, db = sur.conv3x3_backward(x, wt, y if relu else None, dy, need_dx)
    dz = dy * (y > 0) if relu else dy
    _sums_agree(db, dz)
    if need_dx:
        assert torch.equal(dx, sur.conv3x3(dz, sur.flip_transpose(wt, cin, cout)))
    else:
        assert dx is None
    want = sur.conv3x3_wgrad(x, dz, cout)  # the same kernel: its atomics add in any order
    assert float((dw - want).abs().max()) <= 1e-6 * float(want.abs().max())
