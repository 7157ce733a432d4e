"""The two-cell direct kernel where its last CTA holds missing cells: a domain just above the size
that takes it, made of repeated patterns small enough for the one-cell kernel, evolves as its
pattern does, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from tests.capi import CApiSim

pytestmark = pytest.mark.gpu


def _run(counts, reps, storage, kind, tracer):
    d = len(counts)
    tile = lambda a: np.tile(a, list(reps) + [1] * (a.ndim - d))  # noqa: E731
    s = CApiSim([c * r for c, r in zip(counts, reps)], kind, 1 / 0.6, 1 / 0.8, storage=storage,
                path="direct")
    rng = np.random.default_rng(7)
    s.flags[...] = tile(rng.choice([0] * 8 + [1, 6, 14], counts).astype(np.int32))
    s.rho[...] = tile(1 + rng.uniform(-0.02, 0.02, counts).astype(np.float32))
    s.vel[...] = tile(rng.uniform(-0.05, 0.05, list(counts) + [d]).astype(np.float32))
    if tracer == "16":
        assert s.set_tracer_storage(storage) == 0
    if tracer:
        t = s.add_tracer(1 / 0.55)
        s.vals[t][...] = tile(rng.uniform(0, 1, counts).astype(np.float32))
        s.add_coupling(t, 1.0, 0.2, [1e-4, -2e-4, 1e-4][:d])
    s.iterate(6)
    out = [s.populations(), s.rho, s.vel]
    return out + ([s.tracer_populations(0), s.vals[0]] if tracer else [])


# Cells modulo the 256 of a CTA: 3 (no second cells, and threads without a first), 128 (no second
# cells), 200 (some), 255. The kernel starts at 200,000 cells in 2D and 700,000 in 3D.
LINE = {2: 200000, 3: 700000}


@pytest.mark.parametrize("counts,reps", [((11, 449), (1, 41)), ((32, 45), (14, 10)),
                                         ((24, 241), (7, 5)), ((33, 65), (19, 5))])
@pytest.mark.parametrize("storage,tracer", [("f16", ""), ("bf16", "32"), ("f16", "16")])
@pytest.mark.parametrize("kind", [0, 1])
def test_domains_that_end_within_a_cta_2d(counts, reps, storage, tracer, kind):
    _check(counts, reps, storage, kind, tracer)


@pytest.mark.parametrize("counts,reps", [((15, 17, 107), (5, 11, 1)), ((8, 35, 67), (16, 5, 1))])
@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_domains_that_end_within_a_cta_3d(counts, reps, storage):
    _check(counts, reps, storage, 0, "")


def _check(counts, reps, storage, kind, tracer):
    assert np.prod(counts) < LINE[len(counts)] <= np.prod(counts) * np.prod(reps)
    small = _run(counts, [1] * len(counts), storage, kind, tracer)
    large = _run(counts, reps, storage, kind, tracer)
    for a, b in zip(small, large):
        np.testing.assert_array_equal(np.tile(a, list(reps) + [1] * (a.ndim - len(counts))), b)
