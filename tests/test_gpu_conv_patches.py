"""The tcgen05 convolution and weight gradient on images that their 8 x 16
patches do not tile, on one patch and on more patches than a block takes at a
time, with resident and streamed weights: against the float64 oracle."""

import numpy as np
import pytest

import nn_oracle as nno

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32, 1, 8, 8), (32, 32, 3, 20, 12), (96, 32, 1, 33, 17), (32, 96, 2, 18, 23), (64, 192, 1, 40, 24),
          (192, 64, 2, 17, 9), (128, 64, 5, 16, 8), (128, 384, 1, 24, 40), (384, 128, 1, 22, 16), (32, 128, 1, 15, 31),
          (64, 32, 9, 48, 56),
          # boxes shared between interleaved patches, the last with overhang
          (32, 32, 16, 96, 64), (64, 64, 12, 80, 48), (32, 96, 20, 64, 32), (96, 32, 10, 128, 60)]


def _bf16(a, dev):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(dev).to(torch.bfloat16)


@pytest.mark.parametrize("cin,cout,B,H,W", SHAPES, ids=lambda v: str(v))
def test_convolution_and_weight_gradient_on_any_image_size(cin, cout, B, H, W):
    import torch

    from rang import learned

    dev = torch.device("cuda", 0)
    s = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(cin + 3 * cout + H * W)
    x = nno.bf16(rng.standard_normal((B, H, W, cin)))
    w = nno.bf16(rng.standard_normal((cout, 9, cin)) / np.sqrt(9 * cin))
    b = rng.standard_normal(cout).astype(np.float32)
    dz = nno.bf16(rng.standard_normal((B, H, W, cout)))
    xt, wt, dzt = _bf16(x.reshape(-1, cin), dev), _bf16(w, dev), _bf16(dz.reshape(-1, cout), dev)
    bt = torch.from_numpy(b).to(dev)
    pad = torch.full((B * H * W + 64, cout), 7.0, dtype=torch.bfloat16, device=dev)  # rows past the last stay
    learned._call("conv3", xt.data_ptr(), cin, wt.data_ptr(), bt.data_ptr(), pad.data_ptr(), cout, None, 0, B, H, W,
                  cin, cout, 1, 0, s)
    dw = torch.zeros(cout * 9 * cin, dtype=torch.float32, device=dev)
    db = torch.zeros(cout, dtype=torch.float32, device=dev)
    learned._call("conv3_weight_grad", xt.data_ptr(), cin, dzt.data_ptr(), cout, dw.data_ptr(), db.data_ptr(), B, H, W,
                  cin, cout, s)
    assert learned._library().rang_b200_nn_device_status(s) == 0
    out = pad.float().cpu().numpy()
    assert (out[B * H * W:] == 7.0).all()
    ref = np.maximum(nno.conv3(x, w, b.astype(np.float64)), 0.0)
    # One bfloat16 rounding of the output (2^-8 of the value, 2^-7 of the largest).
    assert np.abs(out[:B * H * W].reshape(ref.shape) - ref).max() <= 2.0**-7 * np.abs(ref).max()
    ref = nno.conv3_weight_grad(x, dz)
    # float32 sums of B H W products of bfloat16 values, exact to 2^-24 of the partial sums.
    assert np.abs(dw.cpu().numpy().reshape(ref.shape) - ref).max() <= 1e-5 * np.abs(ref).max()
    ref = dz.reshape(-1, cout).sum(0)
    assert np.abs(db.cpu().numpy() - ref).max() <= 1e-5 * np.abs(dz).reshape(-1, cout).sum(0).max()
