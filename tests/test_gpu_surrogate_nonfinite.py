"""Weight gradients of operands that are not finite (GPU): infinities and NaNs beside the images'
edges and inside them, in the input and in the output gradient.  Every output pixel contributes
its gradient times the tap's input pixel, or times zero where the image has none, and nothing
else, so a tap is finite exactly where the 64-bit sum is.

A finite element: its products are added in FP32, one unit in the last place (2^-23) of the sum
of their magnitudes lost per addition at most, over the output pixels and the partial sums (at
most one per SM).
"""
import pytest

from test_gpu_surrogate_tiles import ULP, _map, _out

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")
# (image, row, column) of the special pixel; negative: from the end
PLACES = [(0, 0, 0), (1, -1, -1), (0, 0, 5), (1, 6, 0), (0, -1, 4), (1, 3, -1), (0, 4, 6)]


def _sums(x, dy, mode):
    """[nout][9][cin] in 64 bits, zero input where a tap has no pixel."""
    import torch
    Ho, Wo = dy.shape[1:3]
    out = []
    for t in range(9):
        iy, oky = _map(mode, Ho, t // 3 - 1, x.shape[1])
        ix, okx = _map(mode, Wo, t % 3 - 1, x.shape[2])
        tap = x[:, torch.as_tensor(iy, device=x.device)][:, :, torch.as_tensor(ix, device=x.device)]
        ok = torch.as_tensor(oky[:, None] & okx[None, :], device=x.device)[None, :, :, None]
        tap = torch.where(ok, tap, torch.zeros_like(tap))
        out.append(torch.stack([(dy[..., n, None] * tap).sum((0, 1, 2)) for n in range(dy.shape[3])]))
    return torch.stack(out, 1)


@pytest.mark.parametrize("mode", [0, 2, 3])
@pytest.mark.parametrize("where", ["x", "dy", "both"])
@pytest.mark.parametrize("size", [(2, 9, 13), (2, 40, 37)])
def test_weight_gradient_nonfinite(mode, where, size):
    import torch
    from hydist import surrogate as S
    lib = S._bind()
    B, H, W = size
    Ho, Wo = _out(mode, H, W, None, None, odd=1)
    g = torch.Generator(device="cuda").manual_seed(mode * 10 + W)
    for cin, ncol, nout in ((48, 48, 20), (16, 16, 3)):
        for k, (b, i, j) in enumerate(PLACES):
            x = torch.randn((B, H, W, cin), generator=g, device="cuda").to(torch.bfloat16)
            dy = torch.randn((B, Ho, Wo, ncol), generator=g, device="cuda").to(torch.bfloat16)
            if where != "dy":
                x[b, i, j, 3] = INF if k % 2 else NAN
                x[b, i, j, 7] = -INF
            if where != "x":
                dy[b, min(i, Ho - 1), min(j, Wo - 1), 1] = -INF if k % 2 else NAN
                dy[b, min(i, Ho - 1), min(j, Wo - 1), 2] = INF
            dw = torch.zeros((nout, 9, cin), device="cuda")
            err = torch.zeros(1, dtype=torch.int32, device="cuda")
            rc = lib.hyd_conv_wgrad(x.data_ptr(), B, H, W, cin, mode, dy.data_ptr(), Ho, Wo, ncol, nout, dw.data_ptr(),
                                    err.data_ptr(), torch.cuda.current_stream().cuda_stream)
            assert rc == 0 and int(err.item()) == 0
            xd, dd = x.double(), dy.double()[..., :nout]
            ref, mag = _sums(xd, dd, mode), _sums(xd.abs(), dd.abs(), mode)
            fin, inf = torch.isfinite(ref), torch.isinf(ref)
            assert bool((~fin).any())
            assert torch.equal(torch.isnan(dw), torch.isnan(ref)), (k, cin)
            assert torch.equal(dw.double()[inf], ref[inf]), (k, cin)
            assert bool(((dw.double() - ref).abs()[fin] <= (B * Ho * Wo + 148) * ULP * mag[fin]).all()), (k, cin)
