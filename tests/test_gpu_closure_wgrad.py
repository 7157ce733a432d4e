"""The layer-2 weight gradient where a CTA takes many tiles: its ring of stages wraps round, both
halves of its tensor memory are used again, and tiles are added up."""

from __future__ import annotations

import pytest

from tests.test_gpu_closure import cl, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

OFF_W2, CHANNELS, ROWS = 1184, 32, 296


@pytest.mark.parametrize("nx,ny,batch", [(131, 700, 3), (523, 129, 3), (64, 64, 80)])
def test_matches_float64_sums_of_its_operands(torch, cl, nx, ny, batch):  # noqa: F811
    """dW2[co][tap][ci] = sum over cells of dz2[p][co] a1[p + tap][ci], from the kernels' own BF16
    dz2 and a1 (tiles are 4 x 64 cells, one CTA an SM: 7 to 9 tiles each on 148 SMs, with ragged
    edges). Products of BF16 are exact in FP32. Within a tile 16 products are added to the
    accumulators, each addition losing at most the last place of what is there, 2^-23: 8.5 x 2^-23 of
    a sum that grows evenly. Some nine tiles are then added in rounded FP32, 9 x 2^-24, and the CTAs
    in float64. Together below 2^-19 of the gradient."""
    g = torch.Generator(device="cuda").manual_seed(nx)
    net = cl.Net(cl.init_params(3), [0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0])
    bufs = cl.Buffers(nx, ny, batch, train=True)
    n = nx * ny * batch
    x = torch.rand(n * 4, generator=g, device="cuda").to(torch.bfloat16)
    bufs.x.copy_(x.view(torch.int16))
    target = torch.rand(n, generator=g, device="cuda")
    flags = torch.zeros(nx * ny, dtype=torch.int32, device="cuda")
    cl.forward(net, bufs, 0)
    cl.loss_and_grad(net, bufs, target, flags, 0)
    torch.cuda.synchronize()
    cl.status()

    # The workspace ends with dz2, dz1 (each padded to 256 bytes) and the CTAs' partial gradients.
    dz_bytes = (n * CHANNELS * 2 + 255) // 256 * 256
    at = bufs.ws.numel() - 2 * dz_bytes - ROWS * cl.NPARAMS * 4
    dz2 = bufs.ws[at : at + n * CHANNELS * 2].view(torch.bfloat16).view(batch, nx, ny, CHANNELS)
    a1 = bufs.a1.view(torch.bfloat16).view(batch, nx, ny, CHANNELS)
    want = torch.zeros(CHANNELS, 9, CHANNELS, dtype=torch.float64, device="cuda")
    for b in range(batch):
        padded = torch.nn.functional.pad(a1[b].double(), (0, 0, 1, 1, 1, 1))
        dz = dz2[b].double().reshape(-1, CHANNELS)
        for t in range(9):
            shifted = padded[t // 3 : t // 3 + nx, t % 3 : t % 3 + ny].reshape(-1, CHANNELS)
            want[:, t] += dz.T @ shifted
    got = bufs.grad[OFF_W2 : OFF_W2 + 9 * CHANNELS * CHANNELS].double().view_as(want)
    assert float((got - want).norm() / want.norm()) < 2.0**-19
    # No tap, row or column on its own is worse by more than its share.
    for dim in range(3):
        rest = tuple(d for d in range(3) if d != dim)
        err, size = (got - want).pow(2).sum(rest).sqrt(), want.pow(2).sum(rest).sqrt()
        assert bool((err < 2.0**-19 * size.clamp_min(float(want.norm()) / 64)).all())
