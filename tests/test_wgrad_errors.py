"""Weight gradients against 64 bits to the error of FP32 sums, at the edges of
the kernel's staging, and that the bound would show a lost 128-pixel run or a
lost pixel of a halo."""
import pytest
import torch

# cin, cout, dilation, planes, rows, columns: the widest halo one load holds,
# the dilations beyond it, runs that end inside a 128-pixel step, more steps
# than stages and fewer
CASES = [(32, 32, 64, 1, 140, 200), (64, 64, 64, 1, 130, 129), (16, 32, 65, 1, 140, 200), (64, 32, 100, 1, 210, 150),
         (16, 16, 66, 2, 150, 257), (32, 64, 1, 1, 1, 1), (64, 64, 2, 1, 3, 127), (32, 16, 1, 3, 61, 257),
         (16, 16, 7, 2, 300, 128), (32, 32, 3, 2, 260, 300), (16, 32, 2, 1, 37, 385)]
# FP16 products are exact in FP32 and their sums of at most 160,000 terms round
# to about 1e-6 of the largest entry; the bound of the small dilations' test
BOUND = 1e-4


def _inputs(cin, cout, dil, P, H, W):
    g = torch.Generator(device="cpu").manual_seed(cin * 100 + cout + dil)
    x = (torch.rand((P, H, W, cin), generator=g) * 2 - 1).half()
    dz = (torch.rand((P, H, W, cout), generator=g) * 2 - 1).half()
    return x, dz


def _reference(x, dz, dil):
    """dw [cout][ky][kx][cin] and db in 64 bits, a tap at a time."""
    P, H, W, cin = x.shape
    cout = dz.shape[3]
    xd, zd = x.double(), dz.double()
    dw = torch.zeros((cout, 3, 3, cin), dtype=torch.float64, device=x.device)
    for ky in range(3):
        for kx in range(3):
            dy, dx = (ky - 1) * dil, (kx - 1) * dil
            ys, xs = slice(max(0, -dy), min(H, H - dy)), slice(max(0, -dx), min(W, W - dx))
            yi, xi = slice(ys.start + dy, ys.stop + dy), slice(xs.start + dx, xs.stop + dx)
            if ys.stop > ys.start and xs.stop > xs.start:
                z, v = zd[:, ys, xs].reshape(-1, cout), xd[:, yi, xi].reshape(-1, cin)
                dw[:, ky, kx] = z.T @ v
    return dw, zd.sum((0, 1, 2))


def _close(got, ref):
    return (got - ref).abs().max().item() < BOUND * ref.abs().max().item()


@pytest.mark.parametrize("case", CASES)
def test_the_bound_shows_what_staging_can_lose(case):
    cin, cout, dil, P, H, W = case
    x, dz = _inputs(*case)
    dw, db = _reference(x, dz, dil)
    # the last run of the last row, the one most often ragged
    lost = dz.clone()
    lost[P - 1, H - 1, (W - 1) // 128 * 128:] = 0
    dw2, db2 = _reference(x, lost, dil)
    assert not _close(dw2, dw) and not _close(db2, db)
    # a run counted twice
    assert not _close(2 * dw - dw2, dw) and not _close(2 * db - db2, db)
    # one pixel of a run's left halo: its products with tap kx = 0
    x0 = (W - 1) // 128 * 128
    if x0 >= dil:
        z, v = dz[0, H // 2, x0].double(), x[0, H // 2, x0 - dil].double()
        dw3 = dw.clone()
        dw3[:, 1, 0] -= z[:, None] * v[None, :]
        assert not _close(dw3, dw)


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_weight_gradients_to_the_error_of_their_sums(gpu_ctx, case):
    import rtrace_b200 as rt
    cin, cout, dil, P, H, W = case
    dev = torch.device("cuda", gpu_ctx.device)
    x, dz = (t.to(dev) for t in _inputs(*case))
    dw, db = torch.zeros((cout, 3, 3, cin), device=dev), torch.zeros(cout, device=dev)
    torch.cuda.synchronize()
    L = rt._capi.lib()
    st = L.rt_debug_conv_wgrad(gpu_ctx.handle, x.data_ptr(), dz.data_ptr(), P, H, W, cin, cout, dil, dw.data_ptr(),
                               db.data_ptr())
    assert st == 0, L.rt_last_error(gpu_ctx.handle)
    ref_w, ref_b = _reference(x, dz, dil)
    assert _close(dw.double(), ref_w), (dw.double() - ref_w).abs().max().item() / ref_w.abs().max().item()
    assert _close(db.double(), ref_b), (db.double() - ref_b).abs().max().item() / ref_b.abs().max().item()
