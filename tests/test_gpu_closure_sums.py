"""The closure's gradients are sums over every cell of a batch: they must not drift with its size."""

from __future__ import annotations

import pytest

from tests.test_gpu_closure import cl, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

# W1, b1, b2, W3, b3 (dW2's sums stay in the tensor cores' accumulators)
PARTS = {"W1": (0, 1152), "b1": (1152, 1184), "b2": (10400, 10432), "W3": (10432, 10720),
         "b3": (10720, 10721)}


@pytest.mark.parametrize("nx,ny", [(128, 512), (61, 515)])
def test_batch_gradient_is_the_mean_of_the_samples(torch, cl, nx, ny):  # noqa: F811
    """The gradient of 32 samples is the mean of 32 gradients of one: dy differs by 2^-5, which
    every product carries exactly. An FP32 sum of L rounded additions is off by about
    2^-24 sqrt(L) / 3 of itself; a chain has some 40 here and is one of thousands that are added in
    float64, so what is left on each side is the result's own rounding, 2^-24: 2^-23 in all."""
    B = 32
    g = torch.Generator(device="cuda").manual_seed(4)
    net = cl.Net(cl.init_params(3), [0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0])
    flags = torch.zeros(nx * ny, dtype=torch.int32, device="cuda")
    x = (1.0 + torch.rand(B, nx * ny * 4, generator=g, device="cuda")).to(torch.bfloat16)
    shift = 1.0 + torch.rand(B, nx * ny, generator=g, device="cuda")

    def gradient(bufs, samples):
        bufs.x.copy_(x[samples].reshape(-1).view(torch.int16))
        cl.forward(net, bufs, 0)
        target = (bufs.y.reshape(-1) - shift[samples].reshape(-1)).contiguous()
        cl.loss_and_grad(net, bufs, target, flags, 0)
        torch.cuda.synchronize()
        return bufs.grad.double()

    got = gradient(cl.Buffers(nx, ny, B, train=True), slice(0, B))
    one = cl.Buffers(nx, ny, 1, train=True)
    want = sum(gradient(one, slice(b, b + 1)) for b in range(B)) / B
    for name, (i, j) in PARTS.items():
        err = float((got[i:j] - want[i:j]).norm() / want[i:j].norm())
        assert err < 2.0**-23, (name, err)
