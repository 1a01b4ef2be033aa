"""The bias gradient of a convolution to the error of rounded 32-bit sums."""
import pytest
import torch

# planes, rows, columns, cin, cout, dilation: each channel count, runs that end
# inside a 128-pixel step, fewer runs than blocks and many per block, and a
# dilation whose steps hold a run three times
CASES = [(16, 256, 256, 32, 32, 1), (16, 256, 256, 16, 32, 1), (16, 256, 256, 64, 64, 2), (8, 541, 961, 32, 16, 1),
         (4, 260, 1001, 64, 32, 65), (1, 1, 1, 16, 16, 1), (1, 37, 385, 32, 64, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_bias_gradient_rounds_as_32_bit_sums_do(gpu_ctx, case):
    import rtrace_b200 as rt
    P, H, W, cin, cout, dil = case
    dev = torch.device("cuda", gpu_ctx.device)
    g = torch.Generator(device="cpu").manual_seed(P + H + cout)
    x = torch.rand((P, H, W, cin), generator=g).half().to(dev)
    dz = torch.rand((P, H, W, cout), generator=g).half().to(dev)  # of one sign: rounding errors of one sign add up
    L = rt._capi.lib()
    for sign in (1, -1):
        z = dz * sign
        dw, db = torch.zeros((cout, 3, 3, cin), device=dev), torch.zeros(cout, device=dev)
        torch.cuda.synchronize()
        st = L.rt_debug_conv_wgrad(gpu_ctx.handle, x.data_ptr(), z.data_ptr(), P, H, W, cin, cout, dil, dw.data_ptr(),
                                   db.data_ptr())
        assert st == 0, L.rt_last_error(gpu_ctx.handle)
        ref = z.double().sum((0, 1, 2))
        # up to 16 values are added in 32 bits, 15 roundings of at most 2^-24 of
        # the sum of magnitudes, and the total is rounded once
        assert ((db.double() - ref).abs() <= 16 * 2.0 ** -24 * z.double().abs().sum((0, 1, 2))).all()
