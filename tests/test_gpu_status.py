"""A run's status words as results: a bounded device wait that ran out is a
device error, a non-finite port sample a diverged run, the same for a handle on
its own and for a batch on every path.  No wait is made to run out: the words
are part of a saved state (its last two integers) and are set there.
"""
import struct

import pytest

from conftest import load_package
from test_gpu_one_pass import SHAPES, _problem

pkg = load_package()
from special_topics_b200 import _native as N  # noqa: E402
from special_topics_b200.backend import Batch, Engine  # noqa: E402

pytestmark = pytest.mark.gpu

WAIT, SAMPLE = (N.FDTD_ERR_CUDA, 1 << 30), (N.FDTD_ERR_NONFINITE, 3)


def _with_status(eng, words):
    state = eng.save_state()
    eng.load_state(state[:-8] + struct.pack("ii", *words))


@pytest.mark.parametrize("words", [WAIT, SAMPLE], ids=["wait", "sample"])
@pytest.mark.parametrize("streams,blocks", [(0, (0, 0)), (0, (0, 4)), (2, (0, 0))], ids=["chains", "tiles", "members"])
def test_status_words_mean_the_same_in_a_batch(words, streams, blocks):
    engs = [Engine(_problem(SHAPES[q])[1], "f32-table", dft_block=d) for q, d in zip((0, 6), blocks)]
    try:
        with Batch(engs, streams=streams) as b:
            b.run(5)
            _with_status(engs[1], words)
            with pytest.raises(N.FdtdError) as ei:
                b.run(1)
        assert ei.value.code == words[0] and "batch member 1: " in str(ei.value)
        assert ("step 3" in str(ei.value)) == (words == SAMPLE) and str(1 << 30) not in str(ei.value)
        with pytest.raises(N.FdtdError) as ei:
            engs[1].run(1)
        assert ei.value.code == words[0]
        assert engs[1].status() == words and engs[0].status() == (0, -1)
        engs[0].run(1)
    finally:
        for e in engs:
            e.close()
