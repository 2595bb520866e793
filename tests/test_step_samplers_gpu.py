"""The fixed-point moves and contact positions of the epoch's parallel steps against the host's samplers (glibc doubles)
on whole seeded streams: every value and every draw count equal, over the parameters the fixed point covers up to
their bounds (negative and zero xi among them) and beyond them, where the exact form runs."""

import numpy as np
import pytest

from _harness import host_samplers
from modlefork_gb300 import engine

pytestmark = pytest.mark.gpu

STREAMS, PER = 4096, 2000
SEEDS = np.arange(1, STREAMS + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)


@pytest.mark.parametrize("mean,sd", [(2500.0, 125.0), (4000.0, 200.0), (0.0, 1.0), (1.0, 0.3), (30.0, 30.0),
                                     (2500.0, 1e-6), (524287.0, 16383.9), (524288.0, 100.0), (2500.25, 125.0),
                                     (1000.0, 20000.0)])
def test_moves(mean, sd):
    got, draws = engine.probe_samplers(engine.PROBE_MOVE, SEEDS, PER, mean, sd)
    x, want_draws = host_samplers(engine.PROBE_NORMAL, SEEDS, PER, mean, sd)
    x = np.maximum(0.0, x)
    want = np.floor(x) + (x - np.floor(x) >= 0.5)
    assert np.array_equal(draws, want_draws)
    assert np.array_equal(got, want), np.flatnonzero(got != want)[:5]


@pytest.mark.parametrize("sigma,xi", [(5000.0, 0.001), (5000.0, -0.001), (32767.5, 0.0014), (32767.5, -0.0014),
                                      (7000.0, 0.0), (1000.0, 1e-6), (1000.0, -1e-9), (1e-3, 0.001), (5000.0, 0.01),
                                      (5000.0, -0.2), (40000.0, 0.001)])
def test_positions(sigma, xi):
    got, draws = engine.probe_samplers(engine.PROBE_POSITION, SEEDS, PER, sigma, xi)
    noise, want_draws = host_samplers(engine.PROBE_GEV, SEEDS, PER, sigma, xi)
    x = np.clip(2.0 ** 31 + noise * np.where(np.arange(PER) % 2, 1.0, -1.0), -1.0, 2.0 ** 32)
    assert np.array_equal(draws, want_draws)
    assert np.array_equal(got, np.floor(x)), np.flatnonzero(got != np.floor(x))[:5]
