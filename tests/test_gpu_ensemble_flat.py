"""The flat ensemble kernel (the default shape of small ensembles) against the row-staged kernel and
the tile kernel: the same bits for domains of any size, many of them in one CTA's 128 cells, one
cell short of a CTA and one past it."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SETS = [
    [(1, 1)],
    [(1, 1), (1, 2), (2, 1), (3, 5), (1, 127), (1, 1), (128, 1), (7, 9)] * 3,
    [(1, 129), (2, 512), (512, 2), (40, 31), (17, 64)],
    [(61, 67), (127, 129), (33, 500)],
    [(5, 513), (3, 1000), (20, 7)],  # rows the row-staged kernel does not take
]


def _run(counts, storage, trt, shape):
    from boltzmann_b200.ensemble import Ensemble

    rng = np.random.default_rng(11)
    om = 1.0 / rng.uniform(0.6, 0.9, len(counts))
    ens = Ensemble(counts, omega=om, omega_neg=om * 0.9 if trt else None, storage=storage)
    ens.flags[...] = rng.choice([0] * 10 + [1, 6], ens.n)
    ens.rho[...] = 1 + rng.uniform(-0.02, 0.02, ens.n)
    ens.vel[...] = rng.uniform(-0.05, 0.05, (ens.n, 2))
    ens.set_shape(*shape)
    for mode in ("persistent", "graph"):
        ens.iterate(12, mode=mode)
    return ens.populations(), ens.rho.copy(), ens.vel.copy()


@pytest.mark.parametrize("counts", SETS)
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("trt", [False, True])
def test_flat_rows_and_tiles_agree(counts, storage, trt):
    long_rows = max(b for _, b in counts) > 512
    flat = _run(counts, storage, trt, (128, 0))
    for shape in ((64, 0), (128, 2)) if long_rows else ((0, 0), (0, 1), (64, 0), (128, 2)):
        for a, b in zip(flat, _run(counts, storage, trt, shape)):
            np.testing.assert_array_equal(a, b)
