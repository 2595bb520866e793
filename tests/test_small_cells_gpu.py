"""Cells of few LEFs, around the steps between 1, 2, 4, 8 and 16 worker warps: every epoch against the CPU oracle, in
crowded windows (ties, chains, units piled up at the ends) as in roomy ones; and batched launches, whose block size
follows the largest cell while it is small, against the per-chromosome calls."""

import numpy as np
import pytest

from modlefork_gb300 import engine, genome
from test_gpu_parity import compare_cell, small_genome

pytestmark = pytest.mark.gpu


CASES = [(nl, 20_000_000) for nl in (1, 2, 5, 16, 31, 32, 33, 63, 64, 65, 127, 128, 129, 256, 257)]
# a LEF every 2 kb (fewer than these span a small window from end to end and leave no contact to register)
CASES += [(nl, 2000 * nl + 100_000) for nl in (31, 32, 33, 64, 65, 128, 129, 257)]


@pytest.mark.parametrize("nl,length", CASES)
def test_few_lefs(nl, length):
    cfg = genome.genome_config(num_cells=4, burnin_history_length=20, burnin_smoothing_window_size=5,
                               burnin_target_epochs_for_lef_activation=30, min_burnin_epochs=5, max_burnin_epochs=80,
                               seed=nl)
    chrom, bars = small_genome(cfg, length, 12, seed=nl, occupancy="beta")
    compare_cell(cfg, chrom, bars, nl=nl, target=60 * max(1, nl // 6))


@pytest.mark.parametrize("counts", [(10, 20, 32), (20, 64), (5, 128), (20, 129), (30, 30, 30, 700)])
def test_batches_of_small_cells(counts):
    """One launch over cells of these LEF counts, 40 cells each, equals the calls one by one."""
    cfg = genome.genome_config(num_cells=40, max_burnin_epochs=80, min_burnin_epochs=5, burnin_history_length=20,
                               burnin_smoothing_window_size=5, seed=3)
    with engine.Engine(cfg, 0) as eng:
        tasks, bands, want = [], {}, {}
        for k, nl in enumerate(counts):
            chrom, bars = small_genome(cfg, 800_000 + 100_000 * k, 20, seed=k, occupancy="beta")
            cid = eng.upload_chrom(chrom, bars)
            shape = engine.band_shape(cfg, chrom.simulated_size)
            seeds = np.array([engine.cell_seed(chrom.name, chrom.size, cfg.seed, i) for i in range(40)], dtype=np.uint64)
            targets = np.full(40, 50 + nl, dtype=np.uint64)
            band = np.zeros(shape[0] * shape[1], dtype=np.uint32)
            missed, stats = eng.simulate_cells(cid, seeds, targets, 0, nl, band)
            want[cid] = (band, int(missed), [(s.epochs, s.contacts, s.rng_draws) for s in stats])
            bands[cid] = np.zeros(shape[0] * shape[1], dtype=np.uint32)
            tasks += [(cid, int(s), int(t), 0, nl) for s, t in zip(seeds, targets)]
        missed, stats = eng.simulate_batch(tasks, bands)
        for j, cid in enumerate(sorted(bands)):
            got = [(s.epochs, s.contacts, s.rng_draws) for s in stats[40 * j:40 * j + 40]]
            assert got == want[cid][2] and int(missed[cid]) == want[cid][1]
            assert np.array_equal(bands[cid], want[cid][0])
