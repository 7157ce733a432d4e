"""The closure's training kernels at the edges of their tiles (4 x 64, 8 x 32 and 30 x 64 cells):
one cell short of a tile, one past it, smaller than any, several samples; the same checks and
bounds against the float64 oracle as for the ordinary shapes."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import closure_oracle as co
from tests import test_gpu_closure as base
from tests.test_gpu_closure import cl, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 2), (2, 3, 63), (1, 29, 65), (1, 31, 64), (2, 13, 66), (1, 15, 129), (1, 61, 7),
          (1, 14, 33), (2, 29, 31)]


@pytest.mark.parametrize("B,nx,ny", SHAPES)
def test_layers_at_tile_edges(torch, cl, B, nx, ny):  # noqa: F811
    base.test_forward_layers_match_oracle(torch, cl, B, nx, ny, "tcgen05")


@pytest.mark.parametrize("B,nx,ny", SHAPES)
def test_gradient_at_tile_edges(torch, cl, B, nx, ny):  # noqa: F811
    base.test_loss_and_gradient_match_oracle(torch, cl, B, nx, ny, "tcgen05")


def test_layer3_weight_gradient_keeps_all_bits_of_dy(torch, cl):  # noqa: F811
    """dW3 enters the tensor cores with dy as three BF16 parts. With activations and dy that take
    all of their significant bits, each of the 288 sums of 4,096 products must be a float32 sum's
    distance from float64: 4,096 roundings of 2^-24, at most 2.5e-4 of the products' magnitude and
    far less (2^-24 sqrt(4096) = 4e-6) as a norm. Two parts alone would leave 2^-17 = 8e-6 in each
    product's own error, one part 2^-9; both show against the 2e-6 bound on the mean error."""
    net, bufs, flags, flags_t, params, x, g = base._forward(torch, cl, 1, 64, 64, seed=7)
    rng = np.random.default_rng(3)
    target = rng.normal(size=(1, 64, 64)).astype(np.float32)
    cl.loss_and_grad(net, bufs, torch.tensor(target, device="cuda").reshape(-1), flags_t, 0)
    torch.cuda.synchronize()
    dy = bufs.dy.cpu().numpy().reshape(1, 64, 64).astype(np.float64)
    want = co.backward(params, x, g, dy)[10432:10720]
    got = bufs.grad.cpu().numpy().astype(np.float64)[10432:10720]
    assert base._rel(got, want) < 2e-6
