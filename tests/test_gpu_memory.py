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
from special_topics_b200 import earlystop as ES  # noqa: E402
from special_topics_b200.backend import Batch, Engine  # noqa: E402
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


def test_a_handle_fits_beside_one_that_is_running():
    """The first handle is in one run after another in another thread."""
    steps = 20000
    p, q, keeps, need = _sizes(steps)
    left = keeps + 8 * MB
    assert left < need < left + keeps
    done, ran, errors = threading.Event(), [64], []

    def other(a):
        try:
            while not done.is_set() and ran[0] + 500 <= steps:
                a.run(500)
                ran[0] += 500
        except Exception as e:      # noqa: BLE001
            errors.append(e)

    with Engine(p, "f32-table") as a:
        a.run(64)
        with _only(left):
            t = threading.Thread(target=other, args=(a,))
            t.start()
            try:
                for _ in range(3):
                    with Engine(q, "f32-table") as b:
                        b.run(3)
            finally:
                done.set()
                t.join()
        got = _state(a)
    assert not errors
    with Engine(p, "f32-table") as a:
        a.run(ran[0])
        _assert_same(_state(a), got)


def _dft_block(eng):
    N.check(N.lib().fdtd_ctx_set_dft_block(eng._h, 64))          # 64 steps' samples: some 80 MB


def _network(eng):
    ES.EsNet(out_dim=4, max_batch=256).close()


def _material(eng):
    eng._build_tables_on_device()                                # one byte per cell


@pytest.mark.parametrize("act,left", [(_dft_block, 24 * MB), (_network, 24 * MB), (_material, 2 * MB)],
                         ids=["samples", "network", "material"])
def test_calls_that_need_memory_after_a_run(act, left):
    """What the handle itself keeps is given up too."""
    p = _box(152, 200)
    out = []
    for short in (False, True):
        with Engine(p, "f32-table") as a:
            a.run(64)
            if short:
                with _only(left):
                    act(a)
            else:
                need, _ = _cost(lambda: act(a))
                assert act is not _dft_block or need > left
            a.run(64)
            out.append(_state(a))
    _assert_same(*out)


def test_copies_built_for_a_batch_that_cannot_use_them_are_freed():
    """The second member's copies do not fit, so the batch takes the tile list
    and the first member keeps none."""
    p, q = _box(64, 200), _box(128, 200)
    with Engine(q, "f32-table") as b:
        keeps, _ = _cost(lambda: b.run(64))
    with Engine(p, "f32-table") as a, Engine(q, "f32-table") as b, Batch([a, b]) as batch:
        with _only(keeps):
            held, _ = _cost(lambda: batch.run(128))
            assert batch.profile_kernels(1)["e"] > 0
    with Engine(p, "f32-table") as a:
        kept, _ = _cost(lambda: a.run(128))
    assert held < kept


def test_a_dft_block_that_does_not_fit_leaves_per_step_sums():
    """The old block's buffer is gone by then, so the sums are per step from there."""
    p = _box(128, 200)
    with Engine(p, "f32-table", dft_accumulator="kahan-f32", dft_block=16) as a:
        a.run(64)
        with _only(64 * MB):
            with pytest.raises(N.FdtdError) as ei:
                N.check(N.lib().fdtd_ctx_set_dft_block(a._h, 1024))
            assert ei.value.code == N.FDTD_ERR_OOM
        a.run(64)
        got = _state(a)
    with Engine(p, "f32-table", dft_accumulator="kahan-f32") as a:
        a.run(128)
        _assert_same(_state(a), got)
