"""Float32 sums of the convolution's gradients keep the precision of short chains of
additions, whatever the image's size."""
import pytest

pytestmark = pytest.mark.gpu


def _wgrad_error(sur, n, h, w, cin, cout):
    """Largest relative error of the first 8 output channels' weight gradient for
    positive inputs, against float64."""
    import torch
    import torch.nn.functional as F
    g = torch.Generator(device="cuda").manual_seed(cin + w)
    x = (0.5 + torch.rand((n, h, w, cin), generator=g, device="cuda")).to(torch.bfloat16)
    dy = (0.5 + torch.rand((n, h, w, cout), generator=g, device="cuda")).to(torch.bfloat16)
    got = sur.conv3x3_wgrad(x, dy, cout)[:8, : 9 * cin].double()
    xp = F.pad(x.double(), (0, 0, 1, 1, 1, 1))
    d = dy[..., :8].double().reshape(-1, 8).T
    ref = torch.cat([d @ xp[:, ky:ky + h, kx:kx + w].reshape(-1, cin) for ky in range(3) for kx in range(3)], 1)
    return float(((got - ref).abs() / ref).max())


@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 200, 200, 512, 512), (16, 64, 64, 384, 128), (32, 128, 128, 64, 64),
                                            (1, 300, 32, 512, 512), (3, 150, 33, 512, 256)])
def test_wgrad_chains_stay_short(gpu_lib, n, h, w, cin, cout):
    """Positive terms, so that every lost bit has the same sign.  A chain covers 2048
    pixels at most: the error is that of one such image (the sums it is compared
    with, with room of 2 for its own), and an atomic's rounding per chain on top."""
    from skewengine_gb300 import surrogate as sur
    one = _wgrad_error(sur, 1, 32, 64, cin, cout)
    segments = n * h * -(-w // (64 if w > 32 else 32))
    chains = -(-segments * (64 if w > 32 else 32) // 1024)
    assert _wgrad_error(sur, n, h, w, cin, cout) <= 2 * one + chains * 2.0 ** -24


@pytest.mark.parametrize("n,h,w,c", [(2, 256, 256, 32), (16, 32, 32, 256), (1, 37, 41, 256), (3, 131, 129, 64),
                                     (4, 512, 512, 32), (1, 37, 41, 2048)])
def test_bias_gradient_as_close_as_the_tensor_reduction(gpu_lib, n, h, w, c):
    """Root mean square error over the channels of eight gradients of positive terms,
    against float64: no larger than that of the float32 reduction the kernel
    replaces (more pixels than the kernel has threads in all but the third)."""
    import torch
    from skewengine_gb300 import surrogate as sur
    mine = theirs = 0.0
    for seed in range(8):
        g = torch.Generator(device="cuda").manual_seed(seed)
        dy = torch.randn((n, h, w, c), generator=g, device="cuda").abs_().to(torch.bfloat16)
        x = torch.zeros((n, h, w, 8), dtype=torch.bfloat16, device="cuda")
        wt = torch.zeros((c, sur.kpad(8)), dtype=torch.bfloat16, device="cuda")
        ref = dy.double().sum((0, 1, 2))
        db = sur.conv3x3_backward(x, wt, None, dy, need_dx=False)[2]
        mine += float(((db.double() - ref) / ref).pow(2).mean())
        theirs += float(((dy.float().sum((0, 1, 2)).double() - ref) / ref).pow(2).mean())
    assert mine <= theirs
