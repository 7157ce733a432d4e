"""The resident kernel at its limits: a wait that runs out, and calls that take several launches."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tests.capi import _lib, check
from tests.test_gpu_resident import _same, _sim

pytestmark = pytest.mark.gpu

LBM_ERR_CUDA = 3


def _restore(s, tracer, state):
    """The state's own populations and tracer values, from the host."""
    s.upload_populations(state[0])
    if tracer:
        g = np.ascontiguousarray(state[1])
        check(_lib.lbm_upload_g(s.h, 0, C.c_void_p(g.ctypes.data)))
        check(_lib.lbm_upload_tracer(s.h, 0, C.c_void_p(state[2].ctypes.data)))


@pytest.mark.parametrize("counts", [(40, 33), (256, 200)])
@pytest.mark.parametrize("storage,tracer", [("f32", ""), ("f16", "16"), ("f64", "64")])
def test_wait_that_runs_out_is_reported_once_and_recoverable(counts, storage, tracer):
    a = _sim(counts, storage, 1, tracer, "auto")
    b = _sim(counts, storage, 1, tracer, "direct")
    for s in (a, b):
        s.iterate(20)
    state = [a.populations()]
    if tracer:
        state += [a.tracer_populations(0), a.vals[0].copy()]

    # Every wait gives up at once; so it does in the next call, whose words are numbered further.
    check(_lib.lbm_set_spin_limit(a.h, C.c_int64(0)))
    for _ in range(2):
        assert a.raw_iterate(20) == 0
        assert _lib.lbm_synchronize(a.h) == LBM_ERR_CUDA
        assert "status bit 1" in a.last_error() and "neighbours" in a.last_error()
        assert _lib.lbm_synchronize(a.h) == 0  # reported once

    check(_lib.lbm_set_spin_limit(a.h, C.c_int64(-1)))
    for s in (a, b):
        _restore(s, tracer, state)
        s.iterate(20)
    _same(a, b, tracer)
    # A limit that is not reached changes nothing.
    check(_lib.lbm_set_spin_limit(a.h, C.c_int64(1 << 20)))
    for s in (a, b):
        s.iterate(20)
    _same(a, b, tracer)


@pytest.mark.parametrize("tracer", ["", "32"])
def test_a_call_of_several_launches(tracer):
    """More than 4000 steps are several launches, the last of which writes the moments."""
    a = _sim((40, 33), "f32", 1, tracer, "auto")
    b = _sim((40, 33), "f32", 1, tracer, "direct")
    for steps in (8010, 10):
        a.iterate(steps)
        b.iterate(steps)
        _same(a, b, tracer)


@pytest.mark.parametrize("storage,tracer", [("f32", ""), ("f32", "32"), ("f16", "16"), ("bf16", "")])
@pytest.mark.parametrize("kind", [0, 1])
def test_relaxation_field(storage, tracer, kind):
    """A rate per cell, another before each call, as a learned closure sets it."""
    torch = pytest.importorskip("torch")
    counts = (131, 97)
    a = _sim(counts, storage, kind, tracer, "auto")
    b = _sim(counts, storage, kind, tracer, "direct")
    g = torch.Generator(device="cuda").manual_seed(3)
    field = torch.empty(counts, device="cuda")
    for s in (a, b):
        check(_lib.lbm_set_omega_field(s.h, C.c_void_p(field.data_ptr())))
    for _ in range(3):
        field.copy_(1.0 + 0.9 * torch.rand(counts, generator=g, device="cuda"))
        torch.cuda.synchronize()
        for s in (a, b):
            s.iterate(10)
        _same(a, b, tracer)
