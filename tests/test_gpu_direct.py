"""The direct kernels on domains of any size: a periodic pattern repeated over a larger domain must
evolve as the small domain does, bit for bit, whichever kernel each size takes (one cell a thread,
two cells a thread for 16-bit populations on large domains) and wherever rows, tiles and CTAs end."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(counts, reps, storage, collision, tracer, steps=6):
    from boltzmann_b200.core import Simulation, bgk, trt

    dim = len(counts)
    kw = {"tracer_storage": storage} if tracer == "16" else {}
    big = [c * r for c, r in zip(counts, reps)]
    sim = Simulation("gpu", big, bgk(0.7) if collision == "bgk" else trt(0.6, 0.8),
                     storage=storage, **kw)
    rng = np.random.default_rng(5)
    tile = lambda a: np.tile(a, list(reps) + [1] * (a.ndim - dim))  # noqa: E731
    flags = rng.choice([0, 0, 0, 0, 0, 0, 1, 6, 14], counts).astype(np.int32)
    sim.cells.flags[...] = tile(flags)
    sim.fluid.rho[...] = tile(1 + rng.uniform(-0.02, 0.02, counts).astype(np.float32))
    sim.fluid.vel[...] = tile(rng.uniform(-0.05, 0.05, list(counts) + [dim]).astype(np.float32))
    if tracer:
        t = sim.add_tracer("t", bgk(0.6))
        t.val[...] = tile(rng.uniform(0, 1, counts).astype(np.float32))
        sim.add_boussinesq_coupling(t, 1.0, 0.1, np.array([1e-4, -2e-4, 1e-4][:dim], np.float32))
    sim.iterate(steps)
    out = [sim._populations(), np.array(sim.fluid.rho), np.array(sim.fluid.vel)]
    if tracer:
        out += [sim._tracer_populations("t"), np.array(sim.get_tracer("t").val)]
    return out


# Larger domains above and small ones below 151,552 cells, the size from which 16-bit kernels take
# two cells a thread; 151,553 is odd, so its last CTA holds a thread with a missing second cell.
CASES = [
    ((97, 53), (6, 5)),
    ((1, 151), (1151, 1)),
    ((7, 349), (71, 1)),
    ((13, 10, 11), (6, 6, 3)),
    ((5, 7, 61), (3, 8, 3)),
]


@pytest.mark.parametrize("counts,reps", CASES)
@pytest.mark.parametrize("storage,tracer", [("f32", ""), ("f32", "32"), ("f16", ""), ("f16", "32"),
                                            ("f16", "16"), ("bf16", "16"), ("f64", "64")])
@pytest.mark.parametrize("collision", ["bgk", "trt"])
def test_repeated_pattern_evolves_as_one(counts, reps, storage, tracer, collision):
    small = _run(counts, [1] * len(counts), storage, collision, tracer)
    large = _run(counts, reps, storage, collision, tracer)
    for a, b in zip(small, large):
        np.testing.assert_array_equal(np.tile(a, list(reps) + [1] * (a.ndim - len(counts))), b)
