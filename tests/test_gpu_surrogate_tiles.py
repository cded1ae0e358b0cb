"""The convolution kernels where their tiles can go wrong (GPU): images of one pixel, one row
or one column, rows longer than a tile (a tile then holds one run per tap row), sizes just
off the tile and the parity split, batches whose images share a tile, outputs wider or
narrower than the input, and pointers off the 16-byte boundary (weight gradient).

Reference: the layer's sum in 64 bits over the same BF16 operands.  The kernels add the K
products of an element in FP32, at most one unit in the last place (2^-23) lost per
addition, so an element may be off by K 2^-23 times the sum of the products' magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -23


def _map(mode, n, d, size):
    """Input index of every output index 0..n-1 for tap offset d along one axis, and which of
    them exist."""
    o = np.arange(n)
    if mode == 3:
        s = o - d
        i, ok = s // 2, s % 2 == 0
    else:
        i = 2 * o + d if mode == 2 else (o + d if mode == 0 else o - d)
        ok = np.ones(n, bool)
    ok = ok & (i >= 0) & (i < size)
    return np.where(ok, i, 0), ok


def _taps(x, mode, Ho, Wo):
    """[9][B][Ho][Wo][C]: the input pixel of every output pixel and tap, zero outside."""
    import torch
    out = []
    for t in range(9):
        iy, oky = _map(mode, Ho, t // 3 - 1, x.shape[1])
        ix, okx = _map(mode, Wo, t % 3 - 1, x.shape[2])
        g = x[:, torch.as_tensor(iy, device=x.device)][:, :, torch.as_tensor(ix, device=x.device)]
        ok = torch.as_tensor(oky[:, None] & okx[None, :], device=x.device)
        out.append(g * ok[None, :, :, None])
    return torch.stack(out)


SIZES = [  # B, H, W, Ho, Wo (None: the mode's usual size)
    (1, 1, 1, None, None), (2, 3, 1, None, None), (1, 1, 5, None, None), (3, 5, 7, None, None),
    (2, 16, 127, None, None), (1, 3, 600, None, None), (2, 130, 3, None, None), (5, 8, 16, None, None),
    (2, 9, 20, 11, 23), (2, 12, 25, 5, 9),
]


def _out(mode, H, W, Ho, Wo, odd):
    if Ho is not None:
        return Ho, Wo
    return {2: ((H + 1) // 2, (W + 1) // 2), 3: (2 * H - odd, 2 * W - odd)}.get(mode, (H, W))


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("size", SIZES)
def test_conv_tiles(mode, size):
    import torch
    from hydist import surrogate as S
    B, H, W, Ho, Wo = size
    Ho, Wo = _out(mode, H, W, Ho, Wo, odd=1)
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + W)
    net = S.Surrogate()
    for cin, ncol, nout in ((48, 48, 48), (16, 48, 40), (48, 16, 3)):
        x = torch.randn((B, H, W, cin), generator=g, device="cuda").to(torch.bfloat16)
        w = torch.randn((nout, 9, cin), generator=g, device="cuda").to(torch.bfloat16).float()
        b = torch.randn(nout, generator=g, device="cuda")
        wpk = S.pack_weights(w, ncol, cin)
        y = net.conv(x, B, H, W, cin, wpk, b, ncol, nout, mode, False, Ho, Wo, out_f32=True)
        taps = _taps(x.double(), mode, Ho, Wo)
        ref = torch.einsum("tbyxc,ntc->byxn", taps, w.double()) + b.double()
        mag = torch.einsum("tbyxc,ntc->byxn", taps.abs(), w.double().abs()) + b.double().abs()
        assert bool(((y.double() - ref).abs() <= (9 * cin + 1) * ULP * mag).all())
        # BF16 output with ReLU and mask: the FP32 result rounded
        mask = torch.randn((B, Ho, Wo, nout), generator=g, device="cuda").to(torch.bfloat16)
        yb = net.conv(x, B, H, W, cin, wpk, b, ncol, nout, mode, True, Ho, Wo, mask=mask)
        assert torch.equal(yb, (torch.relu(y) * (mask.float() > 0)).to(torch.bfloat16))
    net.check_errors()


@pytest.mark.parametrize("mode", [0, 2, 3])
@pytest.mark.parametrize("size", SIZES)
def test_wgrad_tiles(mode, size):
    import torch
    from hydist import surrogate as S
    B, H, W, Ho, Wo = size
    Ho, Wo = _out(mode, H, W, Ho, Wo, odd=0)
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + W)
    net = S.Surrogate()
    for cin, ncol, nout, shift in ((48, 48, 48, 0), (16, 48, 41, 0), (48, 16, 3, 1), (16, 16, 16, 0)):
        x = torch.randn(B * H * W * cin + shift, generator=g, device="cuda").to(torch.bfloat16)[shift:]
        dy = torch.randn(B * Ho * Wo * ncol + shift, generator=g, device="cuda").to(torch.bfloat16)[shift:]
        dw0 = torch.randn((nout, 9, cin), generator=g, device="cuda")
        dw = dw0.clone()
        rc = net.lib.hyd_conv_wgrad(x.data_ptr(), B, H, W, cin, mode, dy.data_ptr(), Ho, Wo, ncol, nout, dw.data_ptr(),
                                    net.err.data_ptr(), net._stream())
        assert rc == 0
        taps = _taps(x.view(B, H, W, cin).double(), mode, Ho, Wo)
        d = dy.view(B, Ho, Wo, ncol)[..., :nout].double()
        ref = torch.einsum("tbyxc,byxn->ntc", taps, d) + dw0.double()
        mag = torch.einsum("tbyxc,byxn->ntc", taps.abs(), d.abs()) + dw0.double().abs()
        n = B * (Ho + 3) * (Wo + 3) + 32  # additions of one element, the raster's padding included
        assert bool(((dw.double() - ref).abs() <= n * ULP * mag).all())
    net.check_errors()


@pytest.mark.parametrize("npix,ncol,nout,shift", [(1, 48, 48, 0), (33, 16, 3, 0), (70001, 48, 41, 0), (5000, 256, 256, 0),
                                                  (777, 48, 48, 1), (900, 20, 7, 0), (64, 264, 10, 0)])
def test_bias_grad_tiles(npix, ncol, nout, shift):
    """Channel sums over the pixels against 64 bits (npix additions, db added at the end)."""
    import torch
    from hydist import surrogate as S
    g = torch.Generator(device="cuda").manual_seed(npix)
    net = S.Surrogate()
    dy = torch.randn(npix * ncol + shift, generator=g, device="cuda").to(torch.bfloat16)[shift:]
    db0 = torch.randn(nout, generator=g, device="cuda")
    db = db0.clone()
    assert net.lib.hyd_bias_grad(dy.data_ptr(), npix, ncol, nout, db.data_ptr(), net._stream()) == 0
    d = dy.view(npix, ncol)[:, :nout].double()
    ref, mag = d.sum(0) + db0.double(), d.abs().sum(0) + db0.double().abs()
    assert bool(((db.double() - ref).abs() <= (npix + 1) * ULP * mag).all())


@pytest.mark.parametrize("npix,nc,ncol,weighted,shift", [(1, 3, 16, True, 0), (4099, 3, 16, False, 0), (700, 5, 16, True, 0),
                                                         (513, 3, 20, True, 0), (300, 4, 8, True, 0), (300, 3, 16, True, 1)])
def test_mse_grad_tiles(npix, nc, ncol, weighted, shift):
    """The loss against 64 bits and the gradient as the rounded FP32 expression."""
    import torch
    from hydist import surrogate as S
    g = torch.Generator(device="cuda").manual_seed(npix)
    net = S.Surrogate()
    a, b = torch.randn((2, npix, nc), generator=g, device="cuda")
    w = torch.rand(npix, generator=g, device="cuda") if weighted else None
    dy = torch.empty(npix * ncol + shift, dtype=torch.bfloat16, device="cuda")[shift:]
    loss = torch.zeros(1, device="cuda")
    scale = 0.125
    assert net.lib.hyd_mse_grad(a.data_ptr(), b.data_ptr(), w.data_ptr() if weighted else None, npix, nc, ncol, scale,
                                dy.data_ptr(), loss.data_ptr(), net._stream()) == 0
    wt = w[:, None] if weighted else torch.ones((npix, 1), device="cuda")
    want = torch.zeros((npix, ncol), device="cuda")
    want[:, :nc] = 2.0 * wt * (a - b) * scale
    assert torch.equal(dy.view(npix, ncol), want.to(torch.bfloat16))
    ref = (wt.double() * (a.double() - b.double()) ** 2).sum() * scale
    assert abs(float(loss) - float(ref)) <= (npix * nc + 8) * 4 * ULP * float(ref)


@pytest.mark.parametrize("nout,cin,ncol,cinp", [(48, 48, 48, 48), (48, 6, 48, 16), (3, 48, 16, 48), (1, 1, 16, 16)])
def test_pack_matches_the_layout(nout, cin, ncol, cinp):
    """The packing kernel against the layout's formula (pack_index), for weights as they lie
    and for a transposed view."""
    import torch
    from hydist import surrogate as S
    w = torch.randn((nout, 9, cin), generator=torch.Generator().manual_seed(1))
    for v, a, b in ((w, ncol, cinp), (w.permute(2, 1, 0), cinp, ncol)):
        want = S.pack_weights(v, a, b)  # on the CPU: PyTorch
        dev = w.cuda() if v is w else w.cuda().permute(2, 1, 0)
        assert torch.equal(S.pack_weights(dev, a, b).cpu(), want)
