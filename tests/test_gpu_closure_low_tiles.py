"""Layer 3 of the closure's forward pass on its low tiles (small and thin batches) and on its high ones:
the same bits for the same sample."""

from __future__ import annotations

import pytest

from tests.test_gpu_closure import cl, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,batch", [(13, 130, 1), (18, 64, 1), (19, 63, 2), (29, 65, 2), (30, 128, 1),
                                         (31, 129, 1), (61, 200, 1)])
def test_a_sample_alone_and_in_a_large_batch(torch, cl, nx, ny, batch):  # noqa: F811
    """Alone the sample takes low tiles (one turn of the chip); in a batch whose low tiles take more
    than twice the turns of the high ones, those."""

    def turns(rows, n):
        tiles = -(-nx // rows) * -(-ny // 64) * n
        return -(-tiles // 296)

    large = batch
    while turns(6, large) <= 2 * turns(30, large) and large < 4096:
        large *= 2
    assert turns(6, batch) == 1 and turns(6, large) > 2 * turns(30, large)
    net = cl.Net(cl.init_params(3), [0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0])
    g = torch.Generator(device="cuda").manual_seed(nx)
    x = torch.rand(batch * nx * ny * 4, generator=g, device="cuda").to(torch.bfloat16).view(torch.int16)

    def forward(copies):
        bufs = cl.Buffers(nx, ny, batch * copies, train=False)
        bufs.x.copy_(x.repeat(copies))
        cl.forward(net, bufs, 0)
        torch.cuda.synchronize()
        return bufs.y.view(copies, -1)

    one, many = forward(1), forward(large // batch)
    assert torch.isfinite(one).all()
    assert torch.equal(many, one.expand_as(many))
