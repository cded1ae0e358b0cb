"""The bias and loss sums over every pixel (GPU): small whole numbers, whose FP32 sums are exact in
any order, so that a pixel left out or taken twice shows; sizes beyond one turn of the kernels'
grids and off their steps."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npix,ncol,nout,shift", [(31, 48, 48, 0), (4129, 48, 48, 0), (70001, 48, 41, 0),
                                                  (400003, 16, 3, 0), (5000, 256, 256, 0), (70001, 48, 48, 1),
                                                  (900, 20, 7, 0)])
def test_bias_sums_are_exact(npix, ncol, nout, shift):
    import torch
    from hydist import surrogate as S
    lib = S._bind()
    g = torch.Generator(device="cuda").manual_seed(npix)
    dy = torch.randint(1, 5, (npix * ncol + shift,), generator=g, device="cuda").to(torch.bfloat16)[shift:]
    db = torch.full((nout,), 3.0, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert lib.hyd_bias_grad(dy.data_ptr(), npix, ncol, nout, db.data_ptr(), s) == 0
    ref = dy.view(npix, ncol)[:, :nout].double().sum(0) + 3.0
    assert float(ref.max()) < 2 ** 24
    assert torch.equal(db.double(), ref)


@pytest.mark.parametrize("npix", [1, 303104, 303105, 700001])
@pytest.mark.parametrize("nc,ncol,weighted", [(3, 16, True), (3, 16, False), (3, 20, True)])
def test_loss_sum_is_exact(npix, nc, ncol, weighted):
    import torch
    from hydist import surrogate as S
    lib = S._bind()
    g = torch.Generator(device="cuda").manual_seed(npix)
    a = torch.randint(0, 4, (npix, nc), generator=g, device="cuda").float()
    b = torch.randint(0, 4, (npix, nc), generator=g, device="cuda").float()
    w = torch.randint(0, 3, (npix,), generator=g, device="cuda").float() if weighted else None
    dy = torch.empty((npix, ncol), dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(1, device="cuda")
    scale = 0.125
    s = torch.cuda.current_stream().cuda_stream
    assert lib.hyd_mse_grad(a.data_ptr(), b.data_ptr(), w.data_ptr() if weighted else None, npix, nc, ncol, scale,
                            dy.data_ptr(), loss.data_ptr(), s) == 0
    wt = w[:, None] if weighted else torch.ones((npix, 1), device="cuda")
    want = torch.zeros((npix, ncol), device="cuda")
    want[:, :nc] = 2.0 * wt * (a - b) * scale
    assert torch.equal(dy, want.to(torch.bfloat16))
    ref = (wt.double() * (a.double() - b.double()) ** 2).sum()  # in units of the scale
    assert float(ref) < 2 ** 24
    assert float(loss) == float(ref) * scale
