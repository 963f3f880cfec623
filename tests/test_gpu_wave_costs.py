"""Costs of the exact pass that have to grow with the wave and no faster,
measured on the device as ratios within one process (both sides the same
kernel on the same GPU, the best of three passes each)."""
import numpy as np
import pytest
import torch

from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


def _kernel_us(run, kernel, tries=3):
    """Device time of the kernels whose name holds ``kernel`` in one call of ``run``, the best of ``tries``."""
    from torch.profiler import ProfilerActivity, profile

    run()
    best = float("inf")
    for _ in range(tries):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            run()
            torch.cuda.synchronize()
        us = sum(e.device_time_total for e in prof.key_averages() if kernel in e.key)
        assert us > 0.0, kernel
        best = min(best, us)
    return best


def _crowded(P, max_steps, evap_rate=0.01):
    """A pass of one wave whose droplets all start on one cell of a bowl's floor."""
    arr, params = window_world("closed", N=24)
    ep = params.erosion
    ep.max_steps, ep.pit_steps, ep.evap_rate = max_steps, 100000, evap_rate
    g, z, rng = gpu_window(arr), np.zeros(P), np.random.default_rng(5)
    x, y = 12.0 + rng.random(P), 12.0 + rng.random(P)
    return lambda: gm.apply_spawns(g, ep, np.zeros(P, np.int64), x, y, z, z, 1.0, wave=P)


def test_waiting_droplets_do_not_hold_up_the_hand_offs(cuda):
    # four times the droplets on the one cell: four times the hand-offs one after another, and no dearer ones
    few, many = (_kernel_us(_crowded(P, 12), "ordered_apply_kernel") for P in (2048, 8192))
    assert many / few < 5.0, (few, many)


def test_ranks_grow_with_the_entries(cuda):
    # eight times the entries on the same few cells: eight times the slots to rank (sixty-four, if every slot went over
    # the whole of its cell's run)
    short, long_ = (_kernel_us(_crowded(2048, steps, 1e-4), "ordered_rank_kernel") for steps in (100, 800))
    assert long_ / short < 8.0, (short, long_)


def test_lakes_of_one_park_are_walked_together(cuda):
    # a few dozen parks: as many lakes of one park each cost about what one lake of them all does (one after another
    # they took more than four times as long)
    from tests.test_gpu_many_lakes import lake_blocks, spawns

    def walk(cells_a_lake):
        g, ep = lake_blocks(96, cells_a_lake)
        g.lake_room.fill_(1e9)
        sp = spawns(40, 96)
        us = _kernel_us(lambda: gm.apply_spawns(g, ep, *sp, 1.0, wave=40, parks=True), "park_walk_kernel")
        assert int((g.lake_load > 0).sum()) > 20
        return us

    each, one = walk(1), walk(0)
    assert each / one < 2.5, (each, one)
