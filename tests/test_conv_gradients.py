"""Gradient kernels of the surrogate's convolutions: the weight gradient by image
rows (edges of its segments, row chunks and channel blocks) against float64 NumPy,
the ReLU and bias gradient against the tensor expressions it replaces, and the
flipped weights bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sur(gpu_lib):
    from skewengine_gb300 import surrogate
    return surrogate


@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 1, 32, 8), (1, 3, 31, 32, 32), (2, 5, 33, 40, 40), (1, 9, 64, 64, 64),
                                            (3, 4, 65, 96, 32), (1, 17, 100, 72, 72), (2, 33, 32, 128, 136),
                                            (1, 130, 129, 32, 64)])
def test_wgrad_rows_matches_numpy(sur, n, h, w, cin, cout):
    import torch
    rng = np.random.default_rng(cin + cout + w)
    xb = torch.from_numpy(rng.normal(0, 1, (n, h, w, cin)).astype(np.float32)).to(torch.bfloat16)
    db = torch.from_numpy(rng.normal(0, 1, (n, h, w, cout)).astype(np.float32)).to(torch.bfloat16)
    xp = np.pad(xb.double().numpy(), ((0, 0), (1, 1), (1, 1), (0, 0)))
    cols = np.stack([xp[:, ky:ky + h, kx:kx + w, :] for ky in range(3) for kx in range(3)], axis=3)
    ref = db.double().numpy().reshape(-1, cout).T @ cols.reshape(-1, 9 * cin)
    got = sur.conv3x3_wgrad(xb.cuda(), db.cuda(), cout).cpu().double().numpy()
    assert np.all(got[:, 9 * cin:] == 0)
    assert np.abs(got[:, : 9 * cin] - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (2, 7, 9, 32), (1, 33, 45, 64), (3, 16, 16, 256), (1, 5, 5, 2048)])
@pytest.mark.parametrize("relu", [False, True])
def test_relu_grad_equals_tensor_expressions(sur, shape, relu):
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    dy = torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)
    y = torch.randn(shape, generator=g, device="cuda").clamp_min_(0).to(torch.bfloat16)
    if relu:
        y.view(-1)[0] = float("nan")
        dy.view(-1)[-1] = float("inf")
    dz, db = sur.relu_grad(dy, y if relu else None)
    want = dy * (y > 0) if relu else dy
    nan = torch.isnan(want)
    assert torch.equal(nan, torch.isnan(dz))
    assert torch.equal(dz.masked_fill(nan, 0).view(torch.int16), want.masked_fill(nan, 0).view(torch.int16))
    ref = want.double().sum((0, 1, 2))
    # Longest chain of float32 additions: 2 per thread, 256 in a block, 19 + 32 over blocks.
    room = 420 * 2.0 ** -24 * want.double().abs().sum((0, 1, 2))
    fin = torch.isfinite(ref)
    assert torch.equal(fin, torch.isfinite(db))
    assert bool(((db.double() - ref).abs() <= room)[fin].all())
    again = sur.relu_grad(dy, y if relu else None)[1]
    assert torch.equal(again[fin], db[fin])


def test_relu_grad_leaves_other_layouts_alone(sur):
    import torch
    dy = torch.zeros((1, 2, 2, 24), dtype=torch.bfloat16, device="cuda")
    assert sur.relu_grad(dy) is None  # 3 groups of 8 channels do not divide a block
    assert sur.relu_grad(dy[..., :8]) is None
    assert sur.relu_grad(torch.zeros((1, 2, 2, 8), device="cuda")) is None


@pytest.mark.parametrize("cin,cout", [(8, 2), (32, 32), (40, 24), (96, 64)])
def test_flipped_weights(sur, cin, cout):
    import torch
    w = torch.randn((cout, sur.kpad(cin)), device="cuda").to(torch.bfloat16)
    want = torch.zeros((cin, sur.kpad(cout)), dtype=torch.bfloat16, device="cuda")
    want[:, : 9 * cout] = w[:, : 9 * cin].reshape(cout, 9, cin).flip(1).permute(2, 1, 0).reshape(cin, 9 * cout)
    assert torch.equal(sur.flip_transpose(w, cin, cout).view(torch.int16), want.view(torch.int16))
