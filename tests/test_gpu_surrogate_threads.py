"""One layer type called from two host threads with different image sizes (GPU): the calls'
tiles need different amounts of shared memory, and no call may depend on what another thread's
call needs.  Each result is the bits of the same call made alone; weight gradients, whose
additions are not ordered, are sums of small whole numbers, exact in any order.
"""
import threading

import pytest

pytestmark = pytest.mark.gpu

CALLS = 1500


def _work(size, seed):
    """(call, expected) of a forward convolution and a weight gradient of one size."""
    import torch
    from hydist import surrogate as S
    lib = S._bind()
    B, H, W = size
    stream = torch.cuda.Stream()
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(-2, 3, (B, H, W, 48), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randint(-2, 3, (B, H, W, 48), generator=g, device="cuda").to(torch.bfloat16)
    w = S.pack_weights(torch.randn((48, 9, 48), generator=g, device="cuda"), 48, 48)
    y = torch.empty_like(x)
    dw = torch.zeros((48, 9, 48), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s = stream.cuda_stream

    def call():
        rc = lib.hyd_conv_forward(x.data_ptr(), B, H, W, 48, w.data_ptr(), None, 48, 48, 0, 0, None, y.data_ptr(), H, W,
                                  0, err.data_ptr(), s)
        return rc or lib.hyd_conv_wgrad(x.data_ptr(), B, H, W, 48, 0, dy.data_ptr(), H, W, 48, 48, dw.data_ptr(),
                                        err.data_ptr(), s)

    assert call() == 0
    torch.cuda.synchronize()
    return call, stream, (y, y.clone()), (dw, dw.clone()), err


def test_two_threads_two_sizes():
    import torch
    works = [_work((8, 64, 61), 1), _work((1, 8, 7), 2)]  # four tiles a step, and one
    fails = [[], []]

    def loop(k):
        call, stream = works[k][0], works[k][1]
        for n in range(CALLS):
            rc = call()
            if rc:
                fails[k].append((n, rc))
            if n % 64 == 63:
                stream.synchronize()

    ts = [threading.Thread(target=loop, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert fails == [[], []]
    for _, _, (y, y1), (dw, dw1), err in works:
        assert int(err.item()) == 0
        assert torch.equal(y, y1)
        assert torch.equal(dw, dw1 * (CALLS + 1))
