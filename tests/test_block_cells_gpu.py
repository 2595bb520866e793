"""Whole cells at the sizes where the block-parallel epoch steps change shape, every epoch's state against
the CPU oracle: LEF counts around a warp, around the steps between 4, 8 and 16 worker warps, around the
windows of two items per worker thread, and dense ones where units pile up (ties, long chains, many moved
units); barrier counts around a window; per-LEF arrays in shared memory and in global scratch."""

import pytest

from modlefork_gb300 import genome
from test_gpu_parity import compare_cell, small_genome

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 513, 1023, 1024, 1025, 2047, 2049, 3073]


@pytest.mark.parametrize("skip_burnin", [0, 1])
@pytest.mark.parametrize("nl", SIZES)
def test_cell_at_step_edges(nl, skip_burnin):
    cfg = genome.genome_config(num_cells=4, skip_burnin=skip_burnin, burnin_history_length=20,
                               burnin_smoothing_window_size=5, burnin_target_epochs_for_lef_activation=30,
                               min_burnin_epochs=5, max_burnin_epochs=60, seed=nl)
    chrom, bars = small_genome(cfg, 40_000_000, 200, seed=nl, occupancy="beta")
    st = compare_cell(cfg, chrom, bars, nl=nl, target=40 * max(1, nl // 6))
    assert st.contacts > 0


@pytest.mark.parametrize("mode", ["fast", "global_scratch"])
@pytest.mark.parametrize("nl,length", [(300, 300_000), (1100, 1_500_000), (2100, 2_000_000)])
def test_crowded_cell(nl, length, mode):
    """A LEF every kilobase: long chains of stalled units, ties at the barriers and chromosome ends."""
    cfg = genome.genome_config(num_cells=4, skip_burnin=1, seed=nl)
    chrom, bars = small_genome(cfg, length, 30, seed=nl, occupancy="beta")
    compare_cell(cfg, chrom, bars, nl=nl, target=20 * (nl // 6), mode=mode)


@pytest.mark.parametrize("nbarriers", [0, 1, 32, 255, 257, 513, 2049, 4100])
def test_barrier_counts(nbarriers):
    cfg = genome.genome_config(num_cells=4, skip_burnin=1, seed=nbarriers)
    chrom, bars = small_genome(cfg, 10_000_000, nbarriers, seed=nbarriers, occupancy="beta")
    compare_cell(cfg, chrom, bars, nl=260, target=1500)


@pytest.mark.parametrize("nl", [700, 2500])
def test_ties_at_the_chromosome_ends(nl):
    """Units bound in the first epoch pile up at the ends with equal positions and epochs: the ranking's
    order of full ties is the reference's."""
    cfg = genome.genome_config(num_cells=4, skip_burnin=1, seed=nl, avg_lef_processivity=4_000_000)
    chrom, bars = small_genome(cfg, nl * 8000, 20, seed=nl, occupancy="beta")
    compare_cell(cfg, chrom, bars, nl=nl, target=60 * (nl // 6))
