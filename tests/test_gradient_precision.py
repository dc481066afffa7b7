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
