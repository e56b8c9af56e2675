"""GPU tests of the batched forward model on uneven spectra (the
persistent-launch form): every tile (warps per block), schedule and
occupancy, the autotuner and the CUDA-graph replay give the same bits as one
rtb_cirsrtfg_wave call per spectrum, a re-prepared batch of the tuned shape
starts with the tuned configuration, and the batch agrees with the FP64
oracle within the parity tolerances."""
import os

import numpy as np
import pytest

from radtrancode_b200 import cirsradg, synth
from tests.helpers import JAC_TOL, RAD_TOL, jac_err, rad_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def uneven():
    kt, cia, _ = synth.config2()
    jobs = synth.config3_jobs(kt, 24, seed=1003)
    return kt, cia, jobs


def _same(outs, singles):
    for (c, g, gt), (c1, g1, gt1) in zip(outs, singles):
        assert np.array_equal(c, c1) and np.array_equal(g, g1) and np.array_equal(gt, gt1)


def test_schedules_graph_and_autotune_are_bit_identical(ctx, uneven):
    kt, cia, jobs = uneven
    ctx.set_ktables(kt)
    ctx.set_cia(cia)
    singles = [ctx.cirsrtfg_wave(j) for j in jobs]
    ctx.prepare(jobs)
    try:
        for tile in (4, 2, 8):
            ctx.set_tile(tile)
            for sched in (0, 1, 2):
                for occ in (0, 1):
                    ctx.set_schedule(sched, occ)
                    ctx.launch()
                    _same(ctx.fetch(), singles)
        ctx.set_tile(0)
        ctx.use_graph(True)
        for _ in range(3):                       # capture, then two replays
            ctx.launch()
            _same(ctx.fetch(), singles)
        tune = ctx.autotune()
        assert tune["candidates"] >= 9 and tune["ms"] > 0 and tune["warps"] in (2, 4, 8)
        ctx.launch()
        _same(ctx.fetch(), singles)
        assert ctx.stats()["cells"] == sum(j.nlayer * j.nwave for j in jobs)
        # a batch of the same shape starts with the tuned tile: the launch's grid is the tuned one
        grid_tuned = ctx.stats()["grid"]
        ctx.use_graph(False)
        ctx.prepare(jobs[::-1])
        ctx.launch()
        _same(ctx.fetch()[::-1], singles)
        assert ctx.stats()["grid"] == grid_tuned
    finally:
        ctx.use_graph(False)
        ctx.set_tile(0)
        ctx.set_schedule(0, 0)


def test_uneven_batch_against_fp64_oracle(ctx, oracle, uneven):
    """Every spectrum of the 24-spectrum uneven batch (one persistent launch)
    against the FP64 oracle."""
    kt, cia, jobs = uneven
    ctx.set_ktables(kt)
    ctx.set_cia(cia)
    outs = ctx.cirsrtfg_wave_batch(jobs)
    worst_r = worst_j = 0.0
    for j, (c, g, gt) in zip(jobs, outs):
        c64, g64, gt64 = oracle.cirsrtfg_wave(kt, cia, j, oracle.ORC_FP64, nthreads=os.cpu_count() or 1)
        worst_r = max(worst_r, rad_err(c, c64))
        worst_j = max(worst_j, jac_err(g, g64, j.nv))
        assert rad_err(c, c64) <= RAD_TOL
        assert jac_err(g, g64, j.nv) <= JAC_TOL
    print(f"uneven batch of {len(jobs)}: radiance {worst_r:.2e}, Jacobian {worst_j:.2e}")


def _by_one_block_and_as_chosen(ctx, kt, cia, jobs):
    """The batch by 8 warps an item in order, and by a context that chooses."""
    outs = []
    for c, fixed in ((ctx, True), (cirsradg.Context(0), False)):
        c.set_ktables(kt)
        c.set_cia(cia)
        if fixed:
            c.set_tile(8)
            c.set_schedule(0, 0)
        try:
            outs.append(c.cirsrtfg_wave_batch(jobs))
        finally:
            if fixed:
                c.set_tile(0)
    return outs


# one item on a cluster of 8, 4 and 2 blocks of 16 warps, on one of 16, a pair of 8 and one of 8
@pytest.mark.parametrize("nwave", [1, 9, 10, 18, 19, 37, 38, 74, 75, 148, 149, 222, 223])
@pytest.mark.parametrize("nlayer,ng", [(2, 20), (23, 20), (40, 16)])
def test_blocks_that_share_an_item_give_the_same_bits(ctx, nwave, nlayer, ng):
    kt, cia = synth.make_ktables([synth.CH4, synth.C2H6], np_=6, nt=5, ng=ng, nbin=256, seed=ng), synth.make_cia(ng)
    job = synth.make_job(kt, [synth.CH4, synth.C2H6], nlayer=nlayer, seed=nwave, nwave=nwave)
    _same(*_by_one_block_and_as_chosen(ctx, kt, cia, [job]))


# items below and from two a block on: in order, and pulled longest spectrum first
@pytest.mark.parametrize("nwave", [60, 150, 450])
def test_chosen_schedule_of_uneven_spectra_gives_the_same_bits(ctx, nwave):
    kt, cia = synth.make_ktables([synth.CH4, synth.C2H6], np_=6, nt=5, ng=20, nbin=512, seed=3), synth.make_cia(3)
    jobs = [synth.make_job(kt, [synth.CH4, synth.C2H6][:1 + k % 2], nlayer=n, seed=k, nwave=nwave)
            for k, n in enumerate([5, 17, 9])]
    _same(*_by_one_block_and_as_chosen(ctx, kt, cia, jobs))


def test_autotune_of_a_small_batch_keeps_the_chosen_form(ctx):
    """Few items: the form a context chooses by itself is among the candidates."""
    kt, cia = synth.make_ktables([synth.CH4], np_=6, nt=5, ng=20, nbin=64, seed=5), synth.make_cia(5)
    job = synth.make_job(kt, [synth.CH4], nlayer=40, seed=5, nwave=3)
    one, = _by_one_block_and_as_chosen(ctx, kt, cia, [job])[:1]
    c = cirsradg.Context(0)
    c.set_ktables(kt)
    c.set_cia(cia)
    c.prepare([job])
    tune = c.autotune()
    assert tune["candidates"] >= 10 and tune["warps"] in (2, 4, 8, 16)
    c.launch()
    _same(c.fetch(), one)


def test_schedule_and_tile_can_be_left_to_the_batch_again(ctx):
    """set_schedule(-1, 0) after another schedule, and every tile that the
    autotuner reports set by hand, 16 warps with several items a block included."""
    kt, cia = synth.make_ktables([synth.CH4, synth.C2H6], np_=6, nt=5, ng=20, nbin=512, seed=3), synth.make_cia(3)
    jobs = [synth.make_job(kt, [synth.CH4, synth.C2H6][:1 + k % 2], nlayer=n, seed=k, nwave=450)
            for k, n in enumerate([5, 17, 9])]
    with cirsradg.Context(0) as c:
        c.set_ktables(kt)
        c.set_cia(cia)
        c.prepare(jobs)
        c.launch()
        chosen, grid = c.fetch(), c.stats()["grid"]
        c.set_schedule(0, 1)
        c.launch()
        _same(c.fetch(), chosen)
        assert c.stats()["grid"] < grid
        c.set_schedule(-1, 0)
        c.launch()
        _same(c.fetch(), chosen)
        assert c.stats()["grid"] == grid
        for tile in (2, 4, 8, 16):
            c.set_tile(tile)
            c.launch()
            _same(c.fetch(), chosen)
        for schedule in (-2, 3):
            with pytest.raises(cirsradg.RtbError, match="ARG"):
                c.set_schedule(schedule, 0)
        with pytest.raises(cirsradg.RtbError, match="ARG"):
            c.set_tile(32)


# a cluster of 8 and of 2 blocks of 16 warps, one of 16, a pair of 8, one of 8: in a fresh context, whose first launch of the form is captured
@pytest.mark.parametrize("nwave", [1, 60, 100, 150, 230])
def test_first_launch_of_a_form_captured(ctx, nwave):
    kt, cia = synth.make_ktables([synth.CH4, synth.C2H6], np_=6, nt=5, ng=12, nbin=256, seed=12), synth.make_cia(12)
    job = synth.make_job(kt, [synth.CH4, synth.C2H6], nlayer=23, seed=nwave, nwave=nwave)
    ctx.set_ktables(kt)
    ctx.set_cia(cia)
    ctx.set_tile(8)
    ctx.set_schedule(0, 0)
    one = [ctx.cirsrtfg_wave(job)]
    with cirsradg.Context(0) as c:
        c.set_ktables(kt)
        c.set_cia(cia)
        c.use_graph(True)
        c.prepare([job])
        for _ in range(2):                   # capture, then a replay
            c.launch()
            _same(c.fetch(), one)
