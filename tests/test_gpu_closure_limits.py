"""The bounded waits of the closure's training kernels: one that runs out is reported, once, and
training stops on it."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_closure import cl, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

LBM_ERR_STATE = 4


@pytest.fixture
def no_polls(cl):  # noqa: F811
    """Every wait for tensor-core products gives up at once."""

    def off():
        assert cl._lib.lbm_closure_set_spin_limit(-1) == 0

    try:
        assert cl._lib.lbm_closure_set_spin_limit(0) == 0
        yield off
    finally:
        off()


def _step(torch, cl, seed=2):  # noqa: F811
    """Two closures: the forward pass, and loss and gradients, of one batch; and its buffers."""
    nx, ny, B = 61, 130, 3  # ragged edges on both axes
    g = torch.Generator(device="cuda").manual_seed(seed)
    net = cl.Net(cl.init_params(3), [0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0])
    bufs = cl.Buffers(nx, ny, B, train=True)
    x = torch.rand(nx * ny * B * 4, generator=g, device="cuda").to(torch.bfloat16)
    bufs.x.copy_(x.view(torch.int16))
    target = torch.rand(nx * ny * B, generator=g, device="cuda")
    flags = torch.zeros(nx * ny, dtype=torch.int32, device="cuda")

    def forward():
        cl.forward(net, bufs, 0)
        torch.cuda.synchronize()
        return bufs.y.clone()

    def backward():
        cl.loss_and_grad(net, bufs, target, flags, 0)
        torch.cuda.synchronize()
        return bufs.grad.clone()

    return forward, backward


def test_waits_that_run_out_are_reported_once(torch, cl):  # noqa: F811
    forward, backward = _step(torch, cl)
    y, grad = forward(), backward()
    cl.status()
    assert cl._lib.lbm_closure_set_spin_limit(0) == 0
    try:
        for run in (forward, backward):
            run()
            assert cl._lib.lbm_closure_status() == LBM_ERR_STATE
            assert b"gave up waiting" in cl._lib.lbm_last_error()
            assert cl._lib.lbm_closure_status() == 0  # cleared by the query
    finally:
        assert cl._lib.lbm_closure_set_spin_limit(-1) == 0
    assert torch.equal(forward(), y) and torch.equal(backward(), grad)
    cl.status()


def _dataset(torch, cl, cfg, samples=4):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(1)
    shape = (samples, *cfg.coarse)
    return cl.Dataset(1.0 + 1e-3 * torch.rand(shape, generator=g, device="cuda"),
                      0.05 * torch.rand((*shape, 2), generator=g, device="cuda"),
                      1e-3 * torch.rand(shape, generator=g, device="cuda"))


def test_training_stops_on_a_wait_that_ran_out(torch, cl, no_polls):  # noqa: F811
    cfg = cl.Config(fine=(256, 256), radius=8.0, batch=2, iters=3)
    data = _dataset(torch, cl, cfg)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        cl.train(cfg, data)
    no_polls()  # the default limit again
    net, report = cl.train(cfg, data)
    assert report.iters == 3 and np.isfinite([loss for _, loss in report.losses]).all()
    assert torch.isfinite(net.params).all()
