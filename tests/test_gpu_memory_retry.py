"""A handle whose first run finds too little memory for the one-pass step's copies
of the state runs half-steps, and the one-pass step once memory is free again,
alone and as a member of a batch, with the same results."""
import pytest

from conftest import load_package
from test_gpu_memory import MB, _box, _only
from test_gpu_one_pass import _assert_same, _state

pkg = load_package()
from special_topics_b200.backend import Batch, Engine  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_copies_are_built_once_memory_is_free(batch):
    p = _box(128, 2000)          # some 110 MB of copies
    with Engine(p, "f32-table") as a, Engine(_box(64, 2000) if batch else p, "f32-table") as b:
        members = [a, b] if batch else [a]
        target = Batch(members) if batch else a
        with _only(48 * MB):
            target.run(30)
            assert target.profile_kernels(1)["e"] > 0
            target.run(600)
            assert target.profile_kernels(1)["e"] > 0
        target.run(600)          # refused for want of memory half-way, asks again in time
        target.run(100)
        assert target.profile_kernels(1)["e"] == 0
        got = [_state(e) for e in members]
        steps = a.step
        if batch:
            target.close()
        for e, want in zip(members, got):
            with Engine(e.problem, "f32-table") as alone:
                alone.run(steps)
                _assert_same(_state(alone), want)
