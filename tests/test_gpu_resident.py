"""The resident kernel (a whole iterate call of a 2D domain that fits on the chip in one launch)
against single-step launches of the direct kernel: the same bits, whatever the tiles, for every
storage, collision and source it takes, over several calls, with several simulations at once."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from tests.capi import CApiSim

pytestmark = pytest.mark.gpu


def _sim(counts, storage, kind, tracer, path, seed=1, gravity=True):
    s = CApiSim(list(counts), kind, 1 / 0.6, 1 / 0.8, storage=storage, path=path)
    rng = np.random.default_rng(seed)
    s.flags[...] = rng.choice([0] * 12 + [1, 6, 8, 14], counts)
    s.rho[...] = (1 + rng.uniform(-0.02, 0.02, counts)).astype(np.float32)
    s.vel[...] = rng.uniform(-0.05, 0.05, list(counts) + [2]).astype(np.float32)
    if tracer == "16":
        assert s.set_tracer_storage(storage) == 0
    if tracer:
        t = s.add_tracer(1 / 0.55, kind=kind, om_neg=1 / 0.7)
        s.vals[t][...] = rng.uniform(0, 1, counts).astype(np.float32)
        if tracer != "uncoupled":
            s.add_coupling(t, 1.0, 0.2, [1e-4, -2e-4])
    elif gravity:
        s.set_gravity([1e-5, -2e-5])
    return s


def _state(s, tracer):
    out = [s.populations(), s.rho.copy(), s.vel.copy()]
    if tracer:
        out += [s.vals[0].copy(), s.tracer_populations(0)]
    return out


def _same(a, b, tracer):
    for x, y in zip(_state(a, tracer), _state(b, tracer)):
        np.testing.assert_array_equal(x, y)


# Domains of one row, column or cell; rows and columns fewer than, as many as and one more than tiles
# along them; tiles with and without cells taken apart; the halo wrapping round the domain.
SHAPES = [(1, 1), (1, 300), (300, 1), (2, 3), (5, 4), (12, 13), (64, 64), (148, 5), (149, 150),
          (97, 211), (300, 299), (31, 1500)]


@pytest.mark.parametrize("counts", SHAPES)
@pytest.mark.parametrize("storage,tracer", [("f32", ""), ("f32", "32"), ("f32", "uncoupled"),
                                            ("f16", ""), ("f16", "32"), ("f16", "16"),
                                            ("bf16", "16"), ("f64", ""), ("f64", "64")])
@pytest.mark.parametrize("kind", [0, 1])
def test_resident_matches_single_steps(counts, storage, tracer, kind):
    a = _sim(counts, storage, kind, tracer, "auto")
    b = _sim(counts, storage, kind, tracer, "direct")
    for steps in (8, 2, 14):  # a call below the least number of steps between two above it
        a.iterate(steps)
        b.iterate(steps)
    _same(a, b, tracer)


@pytest.mark.parametrize("counts,storage", [((820, 817), "f32"), ((760, 850), "f32"),
                                            ((1130, 1090), "f16"), ((577, 573), "f64")])
def test_largest_domains(counts, storage):
    """Around the largest domain whose tiles fit an SM: the resident kernel or single steps."""
    a = _sim(counts, storage, 1, "", "auto")
    b = _sim(counts, storage, 1, "", "direct")
    for s in (a, b):
        s.iterate(44)
    _same(a, b, "")


def test_tracer_added_between_calls():
    a, b = (_sim((90, 70), "f32", 0, "", p, gravity=False) for p in ("auto", "direct"))
    for s in (a, b):
        s.iterate(10)
        t = s.add_tracer(1 / 0.6)
        s.vals[t][...] = np.linspace(0, 1, 6300, dtype=np.float32).reshape(90, 70)
        s.iterate(12)
    _same(a, b, "32")


def test_simulations_at_once():
    """Several threads, each with its own simulation and stream: cooperative launches take turns."""
    sims = [_sim((100 + 7 * k, 120), "f32", 0, "32", "auto", seed=k) for k in range(4)]
    refs = [_sim((100 + 7 * k, 120), "f32", 0, "32", "direct", seed=k) for k in range(4)]

    def work(s):
        for _ in range(20):
            s.iterate(20)

    threads = [threading.Thread(target=work, args=(s,)) for s in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, r in zip(sims, refs):
        for _ in range(20):
            r.iterate(20)
        _same(s, r, "32")
