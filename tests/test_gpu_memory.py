"""Device memory that a handle keeps for speed alone: the padded copies of its
state.  What fits beside the dense arrays of the other handles is accepted, in
any thread, and whoever gave its copies up goes on with the same results.  The
tests take the rest of the device's memory with one buffer, so that sizes of
some 100 MB decide.
"""
import threading
import time
from contextlib import contextmanager

import pytest
import torch

from conftest import load_package
from test_gpu_one_pass import _assert_same, _state

pkg = load_package()
from special_topics_b200 import _native as N  # noqa: E402
from special_topics_b200 import autotune  # noqa: E402
from special_topics_b200.backend import Engine  # noqa: E402
from special_topics_b200.scenario import build_problem_from_scenario  # noqa: E402
from special_topics_b200.workloads import scaling_box  # noqa: E402

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _box(n, steps):
    return build_problem_from_scenario(scaling_box((n, n, n), seed=3, steps=steps), steps, per_cell=False)


def _free():
    return torch.cuda.mem_get_info()[0]


def _cost(make):
    """Device bytes that `make` takes, and what it made."""
    before = _free()
    made = make()
    return before - _free(), made


@contextmanager
def _only(left):
    """All but `left` bytes of the device's free memory are taken."""
    rest = torch.empty(_free() - left, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del rest
        torch.cuda.empty_cache()


def _sizes(steps):
    """The two boxes, what the first keeps beside its dense arrays after a run,
    and what the second needs to exist."""
    p, q = _box(128, steps), _box(152, 64)
    with Engine(p, "f32-table") as a:
        keeps, _ = _cost(lambda: a.run(64))
    need, b = _cost(lambda: Engine(q, "f32-table"))
    b.close()
    return p, q, keeps, need


def test_settings_beside_another_threads_reclaim():
    """One thread sets a handle's launch shape and steps it, with pauses, while
    another creates and frees handles that fit only without its padded copies."""
    steps = 4000
    p, q, keeps, need = _sizes(steps)
    left = keeps + 8 * MB           # room to build the copies again once the other handle is gone
    assert left < need < left + keeps
    done, made, errors = threading.Event(), [0], []

    def other():
        try:
            for _ in range(200):
                if made[0] >= 6:
                    break
                try:
                    with Engine(q, "f32-table") as b:
                        b.run(3)
                        made[0] += 1
                except N.FdtdError as e:
                    if e.code != N.FDTD_ERR_OOM:      # the first handle was in a call
                        raise
                time.sleep(0.004)
        except Exception as e:      # noqa: BLE001
            errors.append(e)
        finally:
            done.set()

    ran = 0
    with Engine(p, "f32-table") as a:
        a.run(64)
        ran += 64
        with _only(left):
            t = threading.Thread(target=other)
            t.start()
            while not done.is_set() and ran + 64 <= steps - 64:
                for chunk in (4, 8, 16, 8):
                    autotune.set_tiling(a, chunk, 4, 1)
                    a.x_wall = True
                a.run(64)
                ran += 64
                time.sleep(0.004)
            t.join()
        a.run(64)
        ran += 64
        got = _state(a)
    assert not errors and made[0] >= 1
    with Engine(p, "f32-table") as a:
        a.run(ran)
        _assert_same(_state(a), got)
