"""Batches that change their path between runs: one-pass chains where the
members' DFT blocks are of one length, the tile list where they are not, member
kernels where streams are set.  Every path does the same arithmetic, so the
members give the same bits as runs on their own, whichever path took which steps.
"""
import numpy as np
import pytest

from conftest import load_package
from test_gpu_one_pass import SHAPES, _assert_same, _problem, _state

pkg = load_package()
from special_topics_b200 import _native as N  # noqa: E402
from special_topics_b200.backend import Batch, Engine  # noqa: E402

pytestmark = pytest.mark.gpu


def _block(eng, steps):
    N.check(N.lib().fdtd_ctx_set_dft_block(eng._h, steps))


def _pair():
    return [_problem(SHAPES[q])[1] for q in (0, 6)]


def _run(engs, advance):
    """Blocks (0, 4), then (0, 0), then (0, 4) again, six steps each."""
    for block in (4, 0, 4):
        _block(engs[1], block)
        advance(6)


@pytest.mark.parametrize("group,per_launch", [(0, 0), (2, 0), (0, 2)])
def test_a_batch_that_changes_path_launches_what_the_path_needs(group, per_launch):
    """Tile list, chains, and the tile list again with the same lists: the third
    run must not find the second's graphs under its own key."""
    alone = []
    for q, p in enumerate(_pair()):
        with Engine(p, "f32-table") as eng:
            for block in (4, 0, 4):
                _block(eng, block if q else 0)
                eng.run(6)
            alone.append(_state(eng))
    engs = [Engine(p, "f32-table") for p in _pair()]
    try:
        with Batch(engs) as b:
            b.set_tiling(8, 4, 1, group, per_launch=per_launch)
            _run(engs, b.run)
        for w, e in zip(alone, engs):
            _assert_same(w, _state(e))
    finally:
        for e in engs:
            e.close()


@pytest.mark.parametrize("streams", [0, 2])
def test_a_batch_sees_what_its_members_set_between_runs(streams):
    """A member's x wall set between two runs of a batch is the second run's."""
    alone = []
    for p in _pair():
        with Engine(p, "f32-table") as eng:
            eng.run(6)
            eng.x_wall = False
            eng.run(6)
            alone.append(_state(eng))
    engs = [Engine(p, "f32-table") for p in _pair()]
    try:
        with Batch(engs, streams=streams) as b:
            b.run(6)
            for e in engs:
                e.x_wall = False
            b.run(6)
        for w, e in zip(alone, engs):
            _assert_same(w, _state(e))
    finally:
        for e in engs:
            e.close()
