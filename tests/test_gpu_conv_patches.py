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
          # images smaller than a patch, down to one pixel, with more and fewer
          # pixels than one block's
          (32, 32, 1, 1, 1), (128, 64, 80, 1, 1), (64, 128, 3, 2, 2), (128, 128, 5, 4, 4), (32, 64, 2, 7, 5),
          (96, 32, 40, 3, 8), (384, 128, 20, 2, 3),
          # where the mma.sync kernels take over: patches counted and their filling
          (32, 32, 511, 1, 3), (32, 32, 512, 1, 3), (128, 128, 1024, 2, 4), (64, 64, 1023, 4, 4), (64, 64, 1024, 4, 4),
          (32, 128, 1100, 1, 2),
          # the weight gradient's blocks of 32, 64 and 128 output channels
          (128, 128, 32, 16, 8), (128, 128, 130, 16, 8), (128, 128, 600, 8, 8), (32, 64, 390, 9, 8), (32, 64, 400, 9, 8),
          # boxes shared between interleaved patches, the last with overhang
          (32, 32, 16, 96, 64), (64, 64, 12, 80, 48), (32, 96, 20, 64, 32), (96, 32, 10, 128, 60),
          # one patch a block too many for one round
          (32, 32, 162, 16, 8), (128, 128, 81, 16, 16)]


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


@pytest.mark.parametrize("cin,cout,B,H,W", [(32, 32, 16, 96, 64), (64, 64, 12, 80, 48), (32, 96, 20, 64, 32),
                                            (96, 32, 10, 128, 60), (32, 32, 40, 16, 122)])
def test_patches_that_share_boxes_give_the_same_bits(cin, cout, B, H, W):
    import torch

    from rang import learned

    dev = torch.device("cuda", 0)
    s = torch.cuda.current_stream().cuda_stream
    x = torch.randn(B * H * W, cin, device=dev).bfloat16()
    w = torch.randn(cout, 9, cin, device=dev).bfloat16()
    b = torch.randn(cout, device=dev)
    lib = learned._library()
    out = []
    for path in (0, 2):
        y = torch.empty(B * H * W, cout, device=dev, dtype=torch.bfloat16)
        lib.rang_b200_nn_set_conv_path(path)
        try:
            learned._call("conv3", x.data_ptr(), cin, w.data_ptr(), b.data_ptr(), y.data_ptr(), cout, None, 0, B, H, W,
                          cin, cout, 1, 0, s)
        finally:
            assert lib.rang_b200_nn_set_conv_path(0) == path
        out.append(y)
    assert lib.rang_b200_nn_device_status(s) == 0
    assert torch.equal(out[0], out[1])


def _us(f, reps=20):
    import torch

    for _ in range(3):
        f()
    best = float("inf")
    for _ in range(5):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(reps):
            f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / reps * 1e3)
    return best


@pytest.mark.parametrize("cin,cout,B,H,W", [(128, 128, 4096, 1, 1), (384, 128, 4096, 1, 1), (128, 64, 4096, 2, 2)])
def test_many_small_images_cost_their_pixels(cin, cout, B, H, W):
    """Patches of 8 x 16 pixels that hold one to four: the default takes no
    longer than the mma.sync kernels (half as long again is the noise's room;
    all patches took 2.5 to 5 times as long)."""
    import torch

    from rang import learned

    dev = torch.device("cuda", 0)
    s = torch.cuda.current_stream().cuda_stream
    x = torch.randn(B * H * W, cin, device=dev).bfloat16()
    w = torch.randn(cout, 9, cin, device=dev).bfloat16()
    b = torch.zeros(cout, device=dev)
    out = torch.empty(B * H * W, cout, device=dev, dtype=torch.bfloat16)

    def conv():
        learned._call("conv3", x.data_ptr(), cin, w.data_ptr(), b.data_ptr(), out.data_ptr(), cout, None, 0, B, H, W,
                      cin, cout, 1, 0, s)

    lib = learned._library()
    took = _us(conv)
    lib.rang_b200_nn_set_conv_path(1)
    try:
        bare = _us(conv)
    finally:
        lib.rang_b200_nn_set_conv_path(0)
    assert took <= 1.5 * bare, (took, bare)
